"""The resident RK4 kernel with waits between warps (rk4_flow.cuh) at the edges of its range.

Cell counts around a warp (16, 32, 33), the largest with a helper warp (608), the smallest without (609), the
largest a CTA takes (640); and batches larger than the GPU runs at a time, whose steps are cut into slices.
Tolerances are the path's (test_gpu_parity.py): states 1e-10, rows 1e-12; slices change no arithmetic, so a sliced
trajectory equals the same one run alone bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

R111 = np.ones(3) / np.sqrt(3.0)


@pytest.fixture(scope="module")
def api(native):
    from classical_mcmc_spin_b200 import gpu_api
    return gpu_api


def _spins(n, seed):
    from classical_mcmc_spin_b200.states import random_unit_spins
    return random_unit_spins(n, seed).ravel()


@pytest.mark.parametrize("drive", [False, True])
@pytest.mark.parametrize("dims", [(4, 4), (4, 8), (3, 11), (19, 32), (21, 29), (20, 32)])
def test_flow_matches_oracle_at_its_edges(api, oracle, dims, drive):
    from classical_mcmc_spin_b200.lattice import Lattice
    kw = dict(K=-1.0, Gamma=0.25, Gammap=-0.02, Ka=0.1, Kb=-0.05, Kc=0.02, h=0.1) if dims[0] % 2 else {}
    lat = Lattice.kitaev(*dims, 1, **kw)
    o = oracle.OracleLattice.kitaev(*dims, 1, **kw)
    s0 = _spins(lat.lattice_size, 40 + dims[0])
    h = lat.to_gpu()
    assert next(n for _, n, fits in h.variants() if fits).startswith("rk4_flow")     # the default: first that fits
    if drive:
        fin = np.tile(R111, 2)
        api.set_gpu_pulse(h, lat.rotate_pulse(fin, fin), 0.5, 0.5, 0.7, 0.1, 0.6)
        o.set_pulse(fin, 0.1, fin, 0.6, 0.5, 0.5, 0.7)
    rows, fin_o = o.md_rk4(s0, 0.0, 0.995, 0.01, 3, gpu_loop=True)
    api.set_gpu_spins(h, s0)
    _, obs, _ = api.integrate_gpu(h, 0.0, 0.995, 0.01, 3, "rk4", with_states=False)
    assert len(obs) == len(rows)
    assert np.abs(obs - rows[:, 1:11]).max() <= 1e-12
    assert np.abs(api.get_gpu_spins(h) - fin_o).max() <= 1e-10


@pytest.mark.parametrize("dims,B,steps,save", [((24, 24), 301, 97, 3), ((4, 4), 1500, 64, 1), ((19, 32), 151, 40, 50)])
def test_sliced_batch_equals_single_runs(api, dims, B, steps, save):
    from classical_mcmc_spin_b200.lattice import Lattice
    lat = Lattice.kitaev(*dims, 1)
    h = lat.to_gpu()
    states = np.stack([_spins(lat.lattice_size, 900 + b) for b in range(B)])
    fd = lat.rotate_pulse(np.tile(R111, 2), np.tile(R111, 2))
    t1, t2 = np.linspace(0.0, 0.6, B), np.linspace(0.2, 0.9, B)
    kw = dict(T0=-0.1, save_interval=save, d1=fd[:6], d2=fd[6:], width=0.3, freq=0.5)
    obs, fin = api.run_batch(h, states, steps, 0.01, t1=t1, t2=t2, a1=np.full(B, 0.4), a2=np.full(B, 0.3), **kw)
    for b in (0, 1, B // 2, B - 2, B - 1):
        o1, f1 = api.run_batch(h, states[b:b + 1], steps, 0.01, t1=t1[b:b + 1], t2=t2[b:b + 1], a1=np.full(1, 0.4),
                               a2=np.full(1, 0.3), **kw)
        np.testing.assert_array_equal(obs[b], o1[0])
        np.testing.assert_array_equal(fin[b], f1[0])


@pytest.mark.parametrize("drive", [False, True])
@pytest.mark.parametrize("dims", [(3, 11), (19, 32), (20, 32), (24, 27)])
def test_ssprk53_matches_oracle_at_its_edges(api, oracle, dims, drive):
    """SSPRK(5,3) on chip (one warp up to 640 cells) and, for 24x27, in global memory: states to 1e-12 over 40 steps
    (the bound of test_gpu_methods.py), rows to 1e-13 of the oracle's sums of the returned states."""
    import fixed_methods as fm
    from classical_mcmc_spin_b200.lattice import Lattice
    kw = dict(Ka=0.1, Kb=-0.05, Kc=0.02, h=0.1) if dims[0] % 2 else {}
    lat = Lattice.kitaev(*dims, 1, **kw)
    o = oracle.OracleLattice.kitaev(*dims, 1, **kw)
    s0 = _spins(lat.lattice_size, 70 + dims[0])
    h = lat.to_gpu()
    if drive:
        fin = np.tile(R111, 2)
        api.set_gpu_pulse(h, lat.rotate_pulse(fin, fin), 0.5, 0.4, 0.9, 0.2, 0.6)
        o.set_pulse(fin, 0.2, fin, 0.6, 0.5, 0.4, 0.9)
    api.set_gpu_spins(h, s0)
    traj, obs, times = api.integrate_gpu(h, 0.0, 0.79, 0.02, 7, "ssprk53")
    rt, rs = fm.integrate(lambda y, t: o.rhs(y, t), s0, 0.0, 0.79, 0.02, 7, "ssprk53")
    np.testing.assert_array_equal(times, rt)
    assert np.abs(np.stack([s for _, s in traj]) - rs).max() <= 1e-12
    np.testing.assert_array_equal(traj[-1][1], api.get_gpu_spins(h))
    for r, (_, s) in enumerate(traj):
        assert np.abs(obs[r, :9] - o.magnetizations(s)).max() <= 1e-13


@pytest.mark.parametrize("kind,dims", [("kitaev", (25, 25)), ("kitaev", (38, 64)), ("kitaev", (35, 66)), ("pyro", (5, 5, 5)),
                                       ("pyro", (6, 6, 6)), ("pyro", (7, 7, 7)), ("pyro", (5, 8, 8)), ("pyro", (8, 8, 8)),
                                       ("pyro", (4, 4, 4)), ("pyro", (2, 3, 5))])
def test_cluster_flow_and_paired_bonds_match_oracle(api, oracle, kind, dims):
    """Lattices over clusters of 2 and 4 CTAs (slabs that cut cell rows, an uneven last slab, the most cells a slab
    takes) and pyrochlore cells with paired bonds, each with a pulse and a field, three trajectories."""
    from classical_mcmc_spin_b200.lattice import Lattice
    if kind == "kitaev":
        lat, o = Lattice.kitaev(*dims, 1), oracle.OracleLattice.kitaev(*dims, 1)
    else:
        kw = dict(h=0.2, Jzz=1.0, Jpm=0.05, Jpmpm=0.02, cubic=True)
        lat = Lattice.pyrochlore_non_kramer(*dims, field_direction=R111, **kw)
        o = oracle.OracleLattice.pyrochlore_nk(*dims, direction=R111, **kw)
    fin = np.tile(R111, lat.N_atoms)
    fd = lat.rotate_pulse(fin, fin)
    o.set_pulse(fin, 0.1, fin, 0.3, 0.5, 0.2, 0.7)
    h = lat.to_gpu()
    states = np.stack([_spins(lat.lattice_size, 300 + b) for b in range(3)])
    one = np.ones(3)
    obs, out = api.run_batch(h, states, 40, 0.01, T0=0.0, save_interval=3, t1=0.1 * one, t2=0.3 * one, a1=0.5 * one,
                             a2=0.5 * one, d1=fd[:3 * lat.N_atoms], d2=fd[3 * lat.N_atoms:], width=0.2, freq=0.7)
    for b in range(3):
        rows, ref = o.md_rk4(states[b], 0.0, 0.395, 0.01, 3, gpu_loop=True)
        assert len(rows) == obs.shape[1]
        assert np.abs(obs[b] - rows[:, 1:11]).max() <= 1e-12
        assert np.abs(out[b] - ref).max() <= 1e-10


def test_sliced_cluster_batch_equals_single_runs(api):
    from classical_mcmc_spin_b200.lattice import Lattice
    lat = Lattice.kitaev(48, 48, 1)
    h = lat.to_gpu()
    states = np.stack([_spins(lat.lattice_size, 500 + b) for b in range(75)])
    obs, fin = api.run_batch(h, states, 60, 0.01, save_interval=4)
    for b in (0, 36, 37, 74):
        o1, f1 = api.run_batch(h, states[b:b + 1], 60, 0.01, save_interval=4)
        np.testing.assert_array_equal(obs[b], o1[0])
        np.testing.assert_array_equal(fin[b], f1[0])


@pytest.mark.parametrize("dims", [(2, 3, 4), (6, 5, 9), (13, 13, 13)])
def test_unpaired_pyrochlore_bonds(api, dims):
    """Breathing pyrochlore (bonds that leave the cell weaker, so nothing is paired): one CTA, a cluster, streamed;
    against RK4 over the flat tables in numpy, states to 1e-12 over 12 steps."""
    from classical_mcmc_spin_b200.lattice import Lattice
    lat = Lattice.pyrochlore_non_kramer(*dims, h=0.2, field_direction=R111, Jzz=1.0, Jpm=0.05, Jpmpm=0.02)
    N, z, e = lat.lattice_size, lat.num_bi, lat.export()
    part = e["partners"].reshape(N, z)
    J = e["bilinear"].reshape(N, z, 3, 3) * np.where(part // 4 == np.arange(N)[:, None] // 4, 1.0, 0.7)[..., None, None]
    assert (e["counts"] == z).all()
    h = api.create_gpu_lattice_data(N, 3, 4, z, e["field"], e["onsite"], J, part, e["counts"], e["frames"], e["afm"])
    B = e["field"].reshape(N, 3)
    f = lambda y: np.cross(np.einsum("nzij,nzj->ni", J, y[part]) - B, y)
    s0 = _spins(N, 77)
    y, dt = s0.reshape(N, 3).copy(), 0.02
    for _ in range(12):
        k1 = f(y)
        k2 = f(y + 0.5 * dt * k1)
        k3 = f(y + 0.5 * dt * k2)
        k4 = f(y + dt * k3)
        y = y + (dt / 6.0) * (k1 + 2.0 * k2 + 2.0 * k3 + k4)
    api.set_gpu_spins(h, s0)
    _, obs, _ = api.integrate_gpu(h, 0.0, 11.5 * dt, dt, 5, "rk4", with_states=False)
    assert np.abs(api.get_gpu_spins(h) - y.ravel()).max() <= 1e-12
    assert np.abs(obs[-1, 3:6] - y.mean(0)).max() <= 1e-13
