"""Streamed RK4 of more trajectories than one group holds: three groups, the last one shorter, over replayed chunks
and the steps left after them, against the same trajectories run alone (one group, another chunk length)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

R111 = np.ones(3) / np.sqrt(3.0)


@pytest.mark.parametrize("graphs", [True, False])
def test_groups_of_trajectories_equal_single_runs(native, graphs):
    """16^3 primitive pyrochlore cells: four vectors are 1.5 MiB, so about 48 trajectories share 0.6 of L2 and 98 run
    as groups of 33, 33 and 32.  No arithmetic depends on the group: equal bit for bit."""
    from classical_mcmc_spin_b200 import gpu_api as api
    from classical_mcmc_spin_b200.lattice import Lattice
    from classical_mcmc_spin_b200.states import random_unit_spins
    lat = Lattice.pyrochlore_non_kramer(16, 16, 16, h=0.2, field_direction=R111, Jzz=1.0, Jpm=0.05, Jpmpm=0.02)
    h = lat.to_gpu()
    h.set_graphs(graphs)
    assert all(not fits for _, _, fits in h.variants())
    B, steps = 98, 300
    states = np.stack([random_unit_spins(lat.lattice_size, 700 + b).ravel() for b in range(B)])
    fd = lat.rotate_pulse(np.tile(R111, 4), np.tile(R111, 4))
    t1, t2 = np.linspace(0.0, 1.0, B), np.linspace(0.5, 1.5, B)
    kw = dict(T0=-0.1, save_interval=7, d1=fd[:12], d2=fd[12:], width=0.3, freq=0.5)
    obs, fin = api.run_batch(h, states, steps, 0.005, t1=t1, t2=t2, a1=np.full(B, 0.4), a2=np.full(B, 0.3), **kw)
    for b in (0, 32, 33, 65, 66, 97):
        o1, f1 = api.run_batch(h, states[b:b + 1], steps, 0.005, t1=t1[b:b + 1], t2=t2[b:b + 1], a1=np.full(1, 0.4),
                               a2=np.full(1, 0.3), **kw)
        np.testing.assert_array_equal(obs[b], o1[0])
        np.testing.assert_array_equal(fin[b], f1[0])
