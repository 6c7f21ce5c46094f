"""The bounded waits of the resident flow kernels: what a wait that gives up returns, and that a healthy run never
does."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KERNELS = ["rk4_flow<2,3,1> maxt=160", "rk4_cluster_flow<2,3,1> cs=2", "rk4_cluster_flow<2,3,1> cs=4"]


@pytest.fixture(scope="module")
def api(native):
    from classical_mcmc_spin_b200 import gpu_api
    return gpu_api


def _handle(kernel):
    """8x16 honeycomb (32 cells on each of four CTAs) pinned to a kernel, and its initial spins."""
    from classical_mcmc_spin_b200.lattice import Lattice
    from classical_mcmc_spin_b200.states import random_unit_spins
    lat = Lattice.kitaev(8, 16, 1)
    h = lat.to_gpu()
    h.set_variant(next(i for i, name, fits in h.variants() if fits and name.startswith(kernel)))
    return h, random_unit_spins(lat.lattice_size, 5).ravel()


def _short_run(api, h, s0):
    api.set_gpu_spins(h, s0)
    _, obs, _ = api.integrate_gpu(h, 0.0, 0.395, 0.01, 3, "rk4", with_states=False)
    return obs, api.get_gpu_spins(h)


@pytest.mark.parametrize("kernel", KERNELS)
def test_a_wait_that_gives_up_returns_a_status_and_leaves_the_handle_usable(api, native, kernel):
    """A limit of 0 ends the wait for a row 30000 steps away after a few thousand tries: the run skips its other steps
    and returns CMD_ERR_WATCHDOG, every CTA of a cluster staying to the end; the next run is as before."""
    h, s0 = _handle(kernel)
    obs, fin = _short_run(api, h, s0)
    h.set_wait_limit(0)
    with pytest.raises(native.CmdError) as e:
        api.integrate_gpu(h, 0.0, 299.9995, 0.001, 30000, "rk4", with_states=False)
    assert e.value.code == native.CMD_ERR_WATCHDOG
    h.set_wait_limit(1 << 30)
    obs2, fin2 = _short_run(api, h, s0)
    np.testing.assert_array_equal(obs2, obs)
    np.testing.assert_array_equal(fin2, fin)


@pytest.mark.parametrize("kernel,limit,gap", [(k, 10**6, 30000) for k in KERNELS] +
                         [(KERNELS[0], 1 << 30, 900000), (KERNELS[1], 1 << 30, 600000)])
def test_rows_may_lie_further_apart_than_a_wait_may_last(api, kernel, limit, gap):
    """The wait for a row lasts as many steps as the caller saves rows apart (57 ms at 30000 steps, over 1.1 s in the
    last two): the run equals the same one in pieces of one gap, bit for bit."""
    h, s0 = _handle(kernel)
    dt = 1e-4
    h.set_wait_limit(limit)
    api.set_gpu_spins(h, s0)
    _, obs, times = api.integrate_gpu(h, 0.0, (2 * gap - 0.5) * dt, dt, gap, "rk4", with_states=False)
    fin = api.get_gpu_spins(h)
    assert len(times) == 3
    api.set_gpu_spins(h, s0)
    rows = []
    for piece in range(2):
        _, o, _ = api.integrate_gpu(h, 0.0, (gap - 0.5) * dt, dt, gap // 10, "rk4", with_states=False)
        rows += [o[0]] if piece == 0 else []
        rows.append(o[-1])
    np.testing.assert_array_equal(obs, np.stack(rows))
    np.testing.assert_array_equal(fin, api.get_gpu_spins(h))


def _batch(api, native, h, s0, n_steps, save):
    """cmd_run_batch_device of two trajectories on a stream of its own, synchronised; its status says it was enqueued."""
    import ctypes as C
    import torch
    states = torch.from_numpy(np.stack([s0, s0])).cuda()
    obs = torch.zeros((2, native.lib().cmd_batch_rows(n_steps, save), 10), dtype=torch.float64, device="cuda")
    d = native.BatchDesc()
    d.B, d.states, d.method, d.width, d.dt = 2, states.data_ptr(), native.CMD_RK4, 1.0, 1e-3
    d.n_steps, d.save_interval, d.obs = n_steps, save, obs.data_ptr()
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    native.check(native.lib().cmd_run_batch_device(h.ptr, C.byref(d), C.c_void_p(st.cuda_stream), None), "batch")
    st.synchronize()


def test_a_long_host_batch_reports_a_wait_that_gave_up(api, native):
    """Time chunks (4096 steps or more) synchronise by themselves."""
    h, s0 = _handle(KERNELS[0])
    st = np.stack([s0, s0])
    good = api.run_batch(h, st, 5000, 1e-3, save_interval=500)
    h.set_wait_limit(0)
    with pytest.raises(native.CmdError) as e:
        api.run_batch(h, st, 320000, 1e-3, save_interval=20000)
    assert e.value.code == native.CMD_ERR_WATCHDOG
    h.set_wait_limit(1 << 30)
    for a, b in zip(api.run_batch(h, st, 5000, 1e-3, save_interval=500), good):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("entry", ["status", "get_spins", "integrate", "batch", "chunked", "observables"])
def test_an_asynchronous_calls_fault_is_reported_once(api, native, entry):
    h, s0 = _handle(KERNELS[0])
    api.set_gpu_spins(h, s0)
    call = {"status": h.run_status, "get_spins": lambda: api.get_gpu_spins(h), "observables": lambda: api.observables_gpu(h),
            "integrate": lambda: api.integrate_gpu(h, 0.0, 0.095, 0.01, 5, "rk4", with_states=False),
            "batch": lambda: api.run_batch(h, s0[None], 10, 0.01), "chunked": lambda: api.run_batch(h, s0[None], 4096, 0.01)}[entry]
    call()
    h.set_wait_limit(0)
    _batch(api, native, h, s0, 60000, 20000)
    h.set_wait_limit(1 << 30)
    with pytest.raises(native.CmdError) as e:
        call()
    assert e.value.code == native.CMD_ERR_WATCHDOG
    call()
    _batch(api, native, h, s0, 100, 10)
    h.run_status()
