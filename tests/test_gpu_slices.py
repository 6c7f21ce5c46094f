"""When a batch is cut into slices of steps, by its launches: rows and kernels launch twice unsliced (the run and the
row finisher), more often sliced."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fn", ["cmd_run_batch_device", "cmd_run_batch_device_noalloc"])
def test_slices_are_used_where_the_final_states_may_hold_them(native, fn):
    """Final states apart from the one initial state: sliced.  No final states, or ones whose memory the initial state
    overlaps (inside it, from below, at its end): whole waves."""
    import torch
    from classical_mcmc_spin_b200.lattice import Lattice
    from classical_mcmc_spin_b200.states import random_unit_spins
    lat = Lattice.kitaev(24, 24, 1)
    h = lat.to_gpu()
    B, n3, n = 301, 3 * lat.lattice_size, 40
    buf = torch.zeros((B + 2) * n3, dtype=torch.float64, device="cuda")
    spins = torch.from_numpy(random_unit_spins(lat.lattice_size, 3).ravel()).cuda()
    obs = torch.zeros((B, n + 1, 10), dtype=torch.float64, device="cuda")
    stream = torch.cuda.Stream()

    def launches(start, final):
        """Offsets in doubles of the shared initial state and of the final states (None: none) in buf."""
        buf[start:start + n3] = spins
        d = native.BatchDesc()
        d.B, d.states, d.shared_initial, d.method, d.width, d.dt = B, buf.data_ptr() + 8 * start, 1, native.CMD_RK4, 1.0, 0.01
        d.n_steps, d.save_interval, d.obs = n, 1, obs.data_ptr()
        d.final_states = None if final is None else buf.data_ptr() + 8 * final
        c = C.c_int32()
        torch.cuda.synchronize()
        native.check(getattr(native.lib(), fn)(h.ptr, C.byref(d), C.c_void_p(stream.cuda_stream), C.byref(c)), fn)
        stream.synchronize()
        h.run_status()
        return c.value

    assert launches(0, n3) > 2 and launches(B * n3, 0) > 2
    first = obs[0].cpu().numpy()
    assert all(np.array_equal(first, o) for o in obs[1:].cpu().numpy())
    assert launches(0, None) == 2
    assert launches(7 * n3, 0) == 2 and launches(0, n3 - 3) == 2 and launches(B * n3 - 3, 0) == 2 and launches(5, 5) == 2
