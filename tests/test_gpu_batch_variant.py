"""The kernel a batch runs: told by cmd_batch_variant, the same in both device entry points, its tables there from
cmd_create on."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def api(native):
    from classical_mcmc_spin_b200 import gpu_api
    return gpu_api


def _lattice(kind, dims):
    from classical_mcmc_spin_b200.lattice import Lattice
    return Lattice.kitaev(*dims, 1) if kind == "kitaev" else Lattice.pyrochlore_non_kramer(*dims, Jzz=1.0, Jpm=0.05)


def _batch(native, lat, B, n_steps):
    """Buffers and description of an undriven batch on torch's device."""
    import torch
    from classical_mcmc_spin_b200.states import random_unit_spins
    st = torch.from_numpy(np.stack([random_unit_spins(lat.lattice_size, 50 + b).ravel() for b in range(B)])).cuda()
    obs = torch.zeros((B, native.lib().cmd_batch_rows(n_steps, 3), 10), dtype=torch.float64, device="cuda")
    fin = torch.zeros_like(st)
    d = native.BatchDesc()
    d.B, d.states, d.method, d.width, d.dt = B, st.data_ptr(), native.CMD_RK4, 1.0, 0.01
    d.n_steps, d.save_interval, d.obs, d.final_states = n_steps, 3, obs.data_ptr(), fin.data_ptr()
    torch.cuda.synchronize()
    return d, st, obs, fin


def _name(h, i):
    return h.variants()[i][1]


# 2-atom cells around a CTA's most, 4-atom cells with one and two per thread, a lattice where the helper warp goes
@pytest.mark.parametrize("kind,dims,small,large", [("kitaev", (25, 26), 1, 200), ("kitaev", (32, 32), 3, 200),
                                                   ("pyro", (4, 8, 10), 2, 200), ("pyro", (6, 9, 10), 2, 200),
                                                   ("kitaev", (18, 10), 1, 424), ("kitaev", (48, 48), 2, 60)])
def test_both_device_entry_points_run_the_kernel_that_is_told(api, native, kind, dims, small, large):
    import torch
    lat = _lattice(kind, dims)
    h, pinned = lat.to_gpu(), lat.to_gpu()
    stream = torch.cuda.Stream()
    for B in (small, large):
        told = h.batch_variant(B)
        out = []
        for handle, fn in ((h, "cmd_run_batch_device"), (h, "cmd_run_batch_device_noalloc"), (pinned, "cmd_run_batch_device")):
            pinned.set_variant(told)
            d, _st, obs, fin = _batch(native, lat, B, 20)
            launches = C.c_int32()
            native.check(getattr(native.lib(), fn)(handle.ptr, C.byref(d), C.c_void_p(stream.cuda_stream), C.byref(launches)), fn)
            stream.synchronize()
            handle.run_status()
            out.append((launches.value, obs.cpu().numpy(), fin.cpu().numpy()))
        for launches, obs, fin in out[1:]:
            assert launches == out[0][0]
            np.testing.assert_array_equal(obs, out[0][1])
            np.testing.assert_array_equal(fin, out[0][2])
        assert pinned.get_variant() == pinned.batch_variant(1) == pinned.batch_variant(1000) == told
    cells = dims[0] * dims[1] * (dims[2] if kind == "pyro" else 1)
    flips = (640 < cells <= 1024) if kind == "kitaev" else (256 < cells <= 512)
    names = [_name(h, h.batch_variant(B)) for B in (1, 1 << 20)]
    assert names[0].startswith("rk4_cluster_flow") == (flips or cells > 1024 or (kind == "pyro" and cells > 512))
    assert (names[0].split("<")[0] != names[1].split("<")[0]) == flips


def test_a_new_handles_first_batch_can_be_captured(api, native):
    """The tables of the cluster kernel are uploaded by cmd_create: the first undriven batch allocates and copies
    nothing, so a caller may record it into a graph of their own."""
    import torch
    lat = _lattice("kitaev", (27, 31))
    ref = lat.to_gpu()
    d, _st, obs, fin = _batch(native, lat, 4, 20)
    native.check(native.lib().cmd_run_batch_device(ref.ptr, C.byref(d), None, None), "batch")
    torch.cuda.synchronize()
    want = obs.cpu().numpy(), fin.cpu().numpy()
    h = lat.to_gpu()
    assert _name(h, h.batch_variant(4)).startswith("rk4_cluster_flow")
    obs.zero_(), fin.zero_()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=torch.cuda.Stream(), capture_error_mode="global"):
        st = torch.cuda.current_stream().cuda_stream
        rc = native.lib().cmd_run_batch_device(h.ptr, C.byref(d), C.c_void_p(st), None)
    native.check(rc, "captured batch")
    g.replay()
    torch.cuda.synchronize()
    np.testing.assert_array_equal(obs.cpu().numpy(), want[0])
    np.testing.assert_array_equal(fin.cpu().numpy(), want[1])
