"""The work that users of this framework have it do, as measurable cases.

Each case is one call through the public entry points (gpu_api, adjoint,
mixed_gpu_api, or the C ABI's device-resident batch) on seeded inputs.  The
kinds:

  plain    integrate_gpu: one trajectory, host arrays in and out
  batched  integrate_gpu_batched: the reference API's pump-probe delay batch
  scan     cmd_run_batch_device: many trajectories with device-resident data
  uneven   run_uneven: controlled Dormand-Prince over lattices of mixed sizes
  adjoint  adjoint_rk4: loss and coupling gradients of an RK4 trajectory
  mixed    integrate_mixed_gpu: SU(2) / SU(3) lattices of the TmFeO3 shape

``exact`` restates every path in plain torch (float64): lattices, drive,
integrators, step control, observables, and the gradient as the forward-mode
derivative of the discrete map.
"""
import ctypes
import math

import numpy as np
import torch

from classical_mcmc_spin_b200 import _native as nat
from classical_mcmc_spin_b200 import adjoint as adj
from classical_mcmc_spin_b200 import gpu_api
from classical_mcmc_spin_b200 import mixed_gpu_api as mixed
from classical_mcmc_spin_b200.lattice import Lattice

KITAEV = dict(K=-1.0, Gamma=0.25, Gammap=-0.02, J=0.0, h=0.0)
PYRO = dict(Jzz=1.0, Jpm=0.05, Jpmpm=0.02, h=0.2)
R3 = 1.0 / math.sqrt(3.0)


def listed():
    return [
        # The smallest everyday call: one trajectory of the 1152-spin honeycomb, M and E every step.
        dict(name="plain_rk4_kitaev24", kind="plain", lattice="kitaev", L1=24, L2=24, L3=1, steps=1000, dt=0.01,
             method="rk4", save=1, states=False, drive=False),
        # The same call with the reference API's default method, a pulse, and saved states.
        dict(name="plain_ssprk53_kitaev24", kind="plain", lattice="kitaev", L1=24, L2=24, L3=1, steps=400, dt=0.01,
             method="ssprk53", save=40, states=True, drive=True),
        # The reference's own batched call: a delay scan on a small lattice.
        dict(name="batched_kitaev8x8_40", kind="batched", lattice="kitaev", L1=8, L2=8, L3=1, B=40, steps=500,
             dt=0.02, save=2),
        # The 2DCS scan: 256 delays, each pump-only, probe-only and pump + probe, 1152 spins.
        dict(name="scan_kitaev24_768", kind="scan", lattice="kitaev", L1=24, L2=24, L3=1, B=768, steps=2000,
             dt=0.01, save=1, drive=True, shared=True),
        # An ensemble on an odd-sized lattice with its own initial states and thinned rows.
        dict(name="scan_kitaev13x18_201", kind="scan", lattice="kitaev", L1=13, L2=18, L3=1, B=201, steps=1500,
             dt=0.01, save=4, drive=False, shared=False),
        # Forward ensemble of the 48x48 honeycomb, larger than one SM holds.
        dict(name="scan_kitaev48_64", kind="scan", lattice="kitaev", L1=48, L2=48, L3=1, B=64, steps=1000, dt=0.01,
             save=1, drive=False, shared=False),
        # Pyrochlore ensemble on 4^3 conventional cells (1024 spins) in a static field, driven.
        dict(name="scan_pyro4_200", kind="scan", lattice="pyro", L1=4, L2=4, L3=4, B=200, steps=800, dt=0.01,
             save=1, drive=True, shared=True),
        # Pyrochlore on 16^3 conventional cells (65536 spins): state in HBM.
        dict(name="scan_pyro16_32", kind="scan", lattice="pyro", L1=16, L2=16, L3=16, B=32, steps=300, dt=0.005,
             save=1, drive=False, shared=False),
        # 256 controlled trajectories over eight lattice classes at tight tolerance.
        dict(name="uneven_rk45_256", kind="uneven", B=256, max_steps=300, tol=1e-10, T1=100.0, final=False),
        # Five-parameter gradients of 64 trajectories on the 48x48 honeycomb.
        dict(name="adjoint_kitaev48_64", kind="adjoint", lattice="kitaev", L1=48, L2=48, L3=1, B=64, steps=400,
             dt=0.01, every=0),
        # Four-parameter gradients on the 65536-spin pyrochlore.
        dict(name="adjoint_pyro16_8", kind="adjoint", lattice="pyro", L1=16, L2=16, L3=16, B=8, steps=100,
             dt=0.005, every=0),
        # TmFeO3-shaped mixed lattice, 864 + 864 sites, default method, both kinds driven.
        dict(name="mixed_ssprk53_6x6x6", kind="mixed", L1=6, L2=6, L3=6, steps=400, dt=0.005, method="ssprk53",
             save=100),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plain", "plain", "batched", "scan", "scan", "scan", "uneven", "adjoint", "adjoint", "mixed"])
    if kind == "plain":
        lattice = rng.choice(["kitaev", "kitaev", "pyro"])
        L = [_log(rng, 4, 32), _log(rng, 4, 32), 1] if lattice == "kitaev" else [rng.randint(2, 4) for _ in range(3)]
        save = rng.choice([1, 3, 50])
        steps = _log(rng, 100, 1000)
        return dict(kind=kind, lattice=lattice, L1=L[0], L2=L[1], L3=L[2], steps=steps, dt=0.01,
                    method=rng.choice(["rk4", "rk4", "ssprk53"]), save=save, states=save == 50,
                    drive=rng.random() < 0.5)
    if kind == "batched":
        return dict(kind=kind, lattice="kitaev", L1=_log(rng, 4, 24), L2=_log(rng, 4, 24), L3=1,
                    B=_log(rng, 8, 160), steps=_log(rng, 200, 800), dt=0.02, save=rng.choice([1, 2, 5]))
    if kind == "scan":
        shape = rng.choice(["small", "small", "cluster", "pyro", "large"])
        if shape == "small":
            L, lattice = [_log(rng, 4, 24), _log(rng, 4, 24), 1], "kitaev"
        elif shape == "cluster":
            L, lattice = [rng.randint(25, 48), rng.randint(25, 48), 1], "kitaev"
        elif shape == "pyro":
            L, lattice = [rng.randint(2, 8) for _ in range(3)], "pyro"
        else:
            L, lattice = [rng.randint(9, 16) for _ in range(3)], "pyro"
        N = L[0] * L[1] * L[2] * (2 if lattice == "kitaev" else 16)
        B = _log(rng, 4, 32) if shape == "large" else _log(rng, 16, 1000)
        most = 5.0e8 if shape != "large" else 4.0e8
        steps = max(20, min(_log(rng, 300, 2000), int(most / (B * N))))
        return dict(kind=kind, lattice=lattice, L1=L[0], L2=L[1], L3=L[2], B=B, steps=steps, dt=0.01 if shape != "large"
                    else 0.005, save=rng.choice([1, 1, 4, 7]), drive=rng.random() < 0.5, shared=rng.random() < 0.5)
    if kind == "uneven":
        return dict(kind=kind, B=_log(rng, 16, 256), max_steps=_log(rng, 60, 250), tol=rng.choice([1e-8, 1e-10]),
                    T1=100.0, final=rng.random() < 0.5)
    if kind == "adjoint":
        if rng.random() < 0.6:
            return dict(kind=kind, lattice="kitaev", L1=rng.randint(8, 48), L2=rng.randint(8, 48), L3=1,
                        B=_log(rng, 4, 64), steps=_log(rng, 60, 350), dt=0.01, every=rng.choice([0, 0, 37]))
        return dict(kind=kind, lattice="pyro", L1=rng.randint(3, 12), L2=rng.randint(3, 12), L3=rng.randint(3, 12),
                    B=_log(rng, 2, 8), steps=_log(rng, 40, 100), dt=0.005, every=0)
    return dict(kind="mixed", L1=rng.randint(2, 7), L2=rng.randint(2, 7), L3=rng.randint(2, 7),
                steps=_log(rng, 50, 300), dt=0.005, method=rng.choice(["ssprk53", "rk4"]), save=50)


# ------------------------------------------------------------------ inputs, from the seed alone
UNEVEN = [("kitaev", L) for L in (8, 12, 16, 24, 32)] + [("pyro", L) for L in (4, 6, 8)]


def _theta(lattice):
    return dict(KITAEV) if lattice == "kitaev" else dict(PYRO)


def _sites(case):
    return case["L1"] * case["L2"] * case["L3"] * (2 if case["lattice"] == "kitaev" else 16)


def _spins(rng, n):
    s = rng.standard_normal((n, 3))
    return s / np.linalg.norm(s, axis=-1, keepdims=True)


def _zigzag(rng, L1, L2):
    """Zigzag chains along the x bond with a Gaussian tilt: the ordered state a 2DCS scan starts from."""
    s = np.where(np.arange(L1).repeat(L2 * 2) % 2 == 0, R3, -R3)[:, None] * np.ones(3)
    s = s + 0.05 * rng.standard_normal(s.shape)
    return s / np.linalg.norm(s, axis=1, keepdims=True)


def _inputs(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "plain":
        return dict(state=_spins(rng, _sites(case)), pulse=(0.5, 0.5, 1.0, 0.5 + rng.random(), 2.0 + rng.random()))
    if kind == "batched":
        return dict(state=_zigzag(rng, case["L1"], case["L2"]), pulse=(0.5, 0.5, 0.0, 0.0, 0.0),
                    taus=np.sort(8.0 * rng.random(case["B"])))
    if kind == "scan":
        B, N = case["B"], _sites(case)
        if case["shared"] and case["lattice"] == "kitaev":
            states = _zigzag(rng, case["L1"], case["L2"]).reshape(1, N, 3)
        else:
            states = _spins(rng, N * (1 if case["shared"] else B)).reshape(-1, N, 3)
        k = np.arange(B)
        pulses = np.stack([np.zeros(B), 100.0 * (k // 3) / max(1, (B + 2) // 3 - 1) + 0.05 * rng.random(),
                           np.where(k % 3 == 1, 0.0, 0.5), np.where(k % 3 == 0, 0.0, 0.5)], axis=1)
        return dict(states=states, pulses=pulses)
    if kind == "uneven":
        pick = np.random.default_rng(case["B"]).integers(0, len(UNEVEN), size=case["B"])   # the batch's composition
        n = [2 * UNEVEN[p][1] ** 2 if UNEVEN[p][0] == "kitaev" else 16 * UNEVEN[p][1] ** 3 for p in pick]
        return dict(pick=pick, states=[_spins(rng, m) for m in n])
    if kind == "adjoint":
        B, N, S = case["B"], _sites(case), case["steps"]
        return dict(states=_spins(rng, B * N).reshape(B, N, 3), targets=0.05 * rng.standard_normal((B, S + 1, 3)))
    return _mixed_inputs(case, rng)


def _mixed_inputs(case, rng):
    """4 SU(2) + 4 SU(3) atoms per cell: 3x3 bonds to the six neighbour cells, 8x8 along x, and 8x3 / 3x8 between
    each SU(3) atom and the SU(2) atoms of its cell and the next cell along an axis."""
    L = (case["L1"], case["L2"], case["L3"])
    nc, na = L[0] * L[1] * L[2], 4
    xyz = np.stack(np.unravel_index(np.arange(nc), L), axis=1)
    at = lambda off: np.ravel_multi_index(tuple(((xyz + off) % L).T), L)
    E, c = np.eye(3, dtype=int), np.arange(nc)
    J, K = 0.3 * rng.standard_normal((na, 3, 3, 3)), 0.15 * rng.standard_normal((na, 8, 8))
    M = 0.15 * rng.standard_normal((na, 2, na, 8, 3))
    part2, bil2 = np.zeros((nc, na, 6), np.int64), np.zeros((nc, na, 6, 3, 3))
    part3, bil3 = np.zeros((nc, na, 2), np.int64), np.zeros((nc, na, 2, 8, 8))
    mp3, mix3 = np.zeros((nc, na, 8), np.int64), np.zeros((nc, na, 8, 8, 3))
    mp2, mix2 = np.zeros((nc, na, 8), np.int64), np.zeros((nc, na, 8, 3, 8))
    for a in range(na):
        for d in range(3):
            part2[:, a, 2 * d], part2[:, a, 2 * d + 1] = at(E[d]) * na + a, at(-E[d]) * na + a
            bil2[:, a, 2 * d], bil2[:, a, 2 * d + 1] = J[a, d], J[a, d].T
        part3[:, a, 0], part3[:, a, 1] = at(E[0]) * na + a, at(-E[0]) * na + a
        bil3[:, a, 0], bil3[:, a, 1] = K[a], K[a].T
        for o in range(2):
            for b in range(na):
                far = E[a % 3]
                mp3[:, a, o * na + b] = (at(far) if o else c) * na + b
                mix3[:, a, o * na + b] = M[a, o, b]
                mp2[:, b, o * na + a] = (at(-far) if o else c) * na + a
                mix2[:, b, o * na + a] = M[a, o, b].T
    sym = lambda x: (x + np.swapaxes(x, 1, 2)) / 2
    A2, A3 = sym(0.05 * rng.standard_normal((na, 3, 3))), sym(0.05 * rng.standard_normal((na, 8, 8)))
    B2, B3 = 0.1 * rng.standard_normal((na, 3)), 0.1 * rng.standard_normal((na, 8))
    tile = lambda x: np.broadcast_to(x, (nc,) + x.shape)
    n = nc * na
    s2, s3 = rng.standard_normal((n, 3)), rng.standard_normal((n, 8))
    state = np.concatenate([(s / np.linalg.norm(s, axis=1, keepdims=True)).ravel() for s in (s2, s3)])
    return dict(n=n, na=na, field2=tile(B2), onsite2=tile(A2), bil2=bil2, part2=part2, field3=tile(B3),
                onsite3=tile(A3), bil3=bil3, part3=part3, mix2=mix2, mp2=mp2, mix3=mix3, mp3=mp3, state=state,
                drive2=rng.standard_normal((2, na, 3)), drive3=rng.standard_normal((2, na, 8)))


# ------------------------------------------------------------------ prepare and run
def _lattice(name, L1, L2, L3):
    if name == "kitaev":
        return Lattice.kitaev(L1, L2, L3, **KITAEV)
    return Lattice.pyrochlore_non_kramer(L1, L2, L3, field_direction=(R3, R3, R3), cubic=True, **PYRO)


def _pulse_field(lat):
    return lat.rotate_pulse(np.tile([R3] * 3, lat.N_atoms), np.tile([R3] * 3, lat.N_atoms))


def prepare(case, seed):
    x = _inputs(case, seed)
    kind = case["kind"]
    if kind == "uneven":
        handles = {int(p): _lattice(UNEVEN[p][0], UNEVEN[p][1], UNEVEN[p][1], 1 if UNEVEN[p][0] == "kitaev" else
                                    UNEVEN[p][1]).to_gpu() for p in sorted(set(x["pick"].tolist()))}
        specs = [dict(handle=handles[int(p)], state=s, T0=0.0, T1=case["T1"], dt=0.01, max_rows=case["max_steps"] + 2,
                      want_final=case["final"]) for p, s in zip(x["pick"], x["states"])]
        return dict(case=case, handles=handles, specs=specs)
    if kind == "mixed":
        n, na, full = x["n"], x["na"], lambda z: np.full(x["n"], z, np.int64)
        h = mixed.create_gpu_mixed_lattice_data(
            n, 3, na, n, 8, na, 6, 2, 8, 8, x["field2"], x["onsite2"], x["bil2"], x["part2"], full(6), x["field3"],
            x["onsite3"], x["bil3"], x["part3"], full(2), x["mix2"], np.zeros(0), x["mp2"], full(8), x["mix3"],
            x["mp3"], full(8))
        mixed.set_gpu_pulse_SU2(h, x["drive2"], 0.5, 0.5, 1.0, 1.0, 2.0)
        mixed.set_gpu_pulse_SU3(h, x["drive3"], 0.5, 0.5, 1.0, 1.0, 2.0)
        return dict(case=case, handle=h, state=x["state"])
    lat = _lattice(case["lattice"], case["L1"], case["L2"], case["L3"])
    h = lat.to_gpu()
    st = dict(case=case, lat=lat, handle=h, **x)
    if kind == "plain" and case["drive"] or kind == "batched":
        gpu_api.set_gpu_pulse(h, _pulse_field(lat), *x["pulse"])
    if kind == "adjoint":
        build = _adjoint_builder(case)
        st["dparams"] = adj.basis_lattices(build, 5 if case["lattice"] == "kitaev" else 4)
    if kind == "scan":
        dev = torch.device("cuda")
        B, N = case["B"], lat.lattice_size
        rows = int(nat.lib().cmd_batch_rows(case["steps"], case["save"]))
        st.update(states=torch.from_numpy(x["states"]).to(dev), pulses=torch.from_numpy(x["pulses"]).to(dev),
                  obs=torch.zeros((B, rows, 10), dtype=torch.float64, device=dev),
                  final=torch.zeros((B, N, 3), dtype=torch.float64, device=dev), fd=_pulse_field(lat))
        d = nat.BatchDesc()
        d.B, d.states, d.shared_initial, d.method = B, st["states"].data_ptr(), int(case["shared"]), nat.CMD_RK4
        d.width, d.freq, d.T0, d.dt = 0.5, 0.0, -5.0 if case["drive"] else 0.0, case["dt"]
        d.n_steps, d.save_interval = case["steps"], case["save"]
        d.obs, d.final_states = st["obs"].data_ptr(), st["final"].data_ptr()
        if case["drive"]:
            d.d1 = st["fd"].ctypes.data
            d.d2 = st["fd"].ctypes.data + 24 * lat.N_atoms
            d.pulse4 = st["pulses"].data_ptr()
        st["desc"] = d
        torch.cuda.synchronize()
    return st


_streams = []


def _stream():
    """The one stream this program queues its device-resident batches on."""
    if not _streams:
        _streams.append(torch.cuda.Stream())
    return _streams[0].cuda_stream


def _adjoint_builder(case):
    L = (case["L1"], case["L2"])
    if case["lattice"] == "kitaev":
        return lambda th: adj.kitaev_lattice(th, *L)
    return lambda th: adj.pyrochlore_lattice(th, *L, case["L3"], cubic=True)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "scan":
        nat.check(nat.lib().cmd_run_batch_device(state["handle"].ptr, ctypes.byref(state["desc"]),
                                                 ctypes.c_void_p(_stream()), None),
                  "cmd_run_batch_device")
        return [state["obs"], state["final"]]
    if kind == "plain":
        h = state["handle"]
        gpu_api.set_gpu_spins(h, state["state"])
        T1 = (case["steps"] - 0.5) * case["dt"]
        traj, obs, times = gpu_api.integrate_gpu(h, 0.0, T1, case["dt"], case["save"], case["method"],
                                                 with_states=case["states"])
        return [obs, times, gpu_api.get_gpu_spins(h), [s for _, s in traj]]
    if kind == "batched":
        T1 = -4.0 + (case["steps"] - 0.5) * case["dt"]
        r = gpu_api.integrate_gpu_batched(state["handle"], state["state"], state["taus"], None, None, -4.0, T1,
                                          case["dt"], case["save"], "rk4")
        return [r.times, r.mag_data]
    if kind == "uneven":
        out = gpu_api.run_uneven(state["specs"], "rk45", case["tol"], case["tol"], max_steps=case["max_steps"])
        res = [np.concatenate([r for r, _, _ in out]), np.array([s for _, _, s in out])]
        return res + [np.concatenate([f for _, f, _ in out])] if case["final"] else res
    if kind == "adjoint":
        return list(adj.adjoint_rk4(state["handle"], state["dparams"], state["states"], 0.0, case["dt"], case["steps"],
                                    state["targets"], checkpoint_every=case["every"]))
    h = state["handle"]
    mixed.set_gpu_mixed_spins(h, state["state"])
    traj, times = mixed.integrate_mixed_gpu(h, 0.0, (case["steps"] - 0.5) * case["dt"], case["dt"], case["save"],
                                            case["method"])
    return [times, [s for _, s in traj]]


# ------------------------------------------------------------------ work one pass cannot do without
def work(case):
    kind = case["kind"]
    if kind == "uneven":
        x = _inputs(case, 0)
        flops = sum((548.0 if UNEVEN[p][0] == "kitaev" else 872.0) * len(s) for p, s in zip(x["pick"], x["states"]))
        values = sum(3.0 * len(s) for s in x["states"])
        return dict(bytes=8 * (values * (2 if case["final"] else 1) + 11.0 * case["B"] * (case["max_steps"] + 1)),
                    flops=flops * case["max_steps"])
    if kind == "mixed":
        n, stages = 4.0 * case["L1"] * case["L2"] * case["L3"], 4 if case["method"] == "rk4" else 5
        per = 2 * (9 + 54 + 192) + 12 + 2 * (64 + 128 + 192) + 162
        return dict(bytes=8 * 11 * n * (1 + case["steps"] // case["save"] + 1), flops=n * per * stages * case["steps"])
    N, z, B = _sites(case), 3 if case["lattice"] == "kitaev" else 6, case.get("B", 1)
    stages = 5 if case.get("method") == "ssprk53" else 4
    step = stages * (18.0 * z + 9 + 12) + (39 if case.get("drive") else 0)
    rows = -(-case["steps"] // case.get("save", 1)) + 1
    if kind == "adjoint":
        nq = 5 if z == 3 else 4
        return dict(bytes=8.0 * B * (3 * N + 6 * rows), flops=B * N * case["steps"] * (step + 4 * (36 * z + 12 * z * nq + 40)))
    states = (1 if kind != "scan" or case["shared"] else B) + B + (rows if case.get("states") else 0)
    return dict(bytes=8.0 * (3 * N * states + (9 if kind == "batched" else 10) * B * rows),
                flops=float(B) * N * case["steps"] * step)


# ------------------------------------------------------------------ the same in plain torch, 64 bits
_DEV = torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(x):
    return torch.as_tensor(np.ascontiguousarray(x), device=_DEV)


def _kitaev_cell(K, Gamma, Gammap, J, h):
    G, P = Gamma, Gammap
    Jx = np.array([[J + K, P, P], [P, J, G], [P, G, J]])
    Jy = np.array([[J, P, G], [P, J + K, P], [G, P, J]])
    Jz = np.array([[J, G, P], [G, J, P], [P, P, J + K]])
    R = np.array([[6 ** -0.5, -(2 ** -0.5), R3], [6 ** -0.5, 2 ** -0.5, R3], [-2 * 6 ** -0.5, 0, R3]])
    bonds = [(Jx, 0, 1, (0, -1, 0)), (Jy, 0, 1, (1, -1, 0)), (Jz, 0, 1, (0, 0, 0))]
    return bonds, np.tile([0.0, h, 0.0], (2, 1)), np.stack([R, R])


def _pyro_cell(Jzz, Jpm, Jpmpm, h, direction=(R3, R3, R3)):
    def ex(th):
        c, s = 2 * Jpmpm * math.cos(th), 2 * Jpmpm * math.sin(th)
        return np.array([[-2 * Jpm + c, -s, 0], [-s, -2 * Jpm - c, 0], [0, 0, Jzz]])
    x, y, z = ex(2 * math.pi / 3), ex(4 * math.pi / 3), ex(0.0)
    kinds = [(z, 0, 1), (x, 0, 2), (y, 0, 3), (y, 1, 2), (x, 1, 3), (z, 2, 3)]
    offs = [(1, 0, 0), (0, 1, 0), (0, 0, 1), (-1, 1, 0), (-1, 0, 1), (0, 1, -1)]
    bonds = [(m, a, b, (0, 0, 0)) for m, a, b in kinds] + [(m, a, b, o) for (m, a, b), o in zip(kinds, offs)]
    ax = np.array([[-2, 1, 1], [-2, -1, -1], [2, 1, -1], [2, -1, 1]]) / math.sqrt(6)
    ay = np.array([[0, -1, 1], [0, 1, -1], [0, -1, -1], [0, 1, 1]]) / math.sqrt(2)
    az = np.array([[1, 1, 1], [1, -1, -1], [-1, 1, -1], [-1, -1, 1]]) / math.sqrt(3)
    field = np.zeros((4, 3))
    field[:, 2] = h * az @ np.asarray(direction)
    return bonds, field, np.stack([ax, ay, az], axis=2)


class _Model:
    """Cells x atoms of one lattice: per atom class the couplings of its bonds and the partner sites."""

    def __init__(self, name, L1, L2, L3, **theta):
        kitaev = name == "kitaev"
        bonds, field, frames = (_kitaev_cell if kitaev else _pyro_cell)(**theta)
        self.NA = 2 if kitaev else 4
        dims = np.array([L1, L2, L3])
        sub = 1 if kitaev else 4
        cube, q = np.divmod(np.arange(L1 * L2 * L3 * sub), sub)
        xyz = np.stack(np.unravel_index(cube, dims), axis=1)
        fcc = np.array([[0, 0, 0], [0, 1, 1], [1, 0, 1], [1, 1, 0]])     # twice the translations of the cube's cells
        prim = np.array([[0, 1, 1], [1, 0, 1], [1, 1, 0]])
        self.G = len(q)
        slots = [[] for _ in range(self.NA)]
        for M, a, b, off in bonds:
            for src, dst, sign, J in ((a, b, 1, M), (b, a, -1, M.T)):
                o = sign * np.asarray(off)
                if kitaev:
                    cell, qq = xyz + o, 0
                else:
                    pos = 2 * xyz + fcc[q] + o @ prim
                    qq = np.select([(pos % 2 == f).all(1) for f in fcc], range(4))
                    cell = (pos - fcc[qq]) // 2
                idx = np.ravel_multi_index(tuple((cell % dims).T), dims) * sub + qq
                slots[src].append((J, idx * self.NA + dst))
        self.part = [_t(np.stack([s[1] for s in sl], axis=1).ravel()) for sl in slots]
        self.J = [_t(np.concatenate([s[0].T for s in sl])) for sl in slots]      # [(3 z), 3]
        self.B, self.frames = _t(field), _t(frames)

    def linear(self, S):
        """sum_n J_n S_p(n) for S [B, G, NA, 3]."""
        flat = S.reshape(S.shape[0], -1, 3)
        H = [flat[:, p].reshape(S.shape[0], self.G, -1) @ J for p, J in zip(self.part, self.J)]
        return torch.stack(H, dim=2)

    def field(self, S):
        return self.linear(S) - self.B

    def rows(self, S):
        """{M_af, M_local, M_global, E/N} of S [B, G, NA, 3]."""
        n = self.G * self.NA
        m = S.sum(1)
        ml, mg = m.sum(1), torch.einsum("aij,baj->bi", self.frames, m)
        e = 0.5 * (S * (self.field(S) - self.B)).sum((1, 2, 3))
        return torch.cat([mg, ml, mg, e[:, None]], 1) / n


def _model(case):
    return _Model(case["lattice"], case["L1"], case["L2"], case["L3"], **_theta(case["lattice"]))


def _rk4_step(f, y, t, dt):
    k1 = f(y, t)
    k2 = f(y + 0.5 * dt * k1, t + 0.5 * dt)
    k3 = f(y + 0.5 * dt * k2, t + 0.5 * dt)
    k4 = f(y + dt * k3, t + dt)
    return y + (dt / 6.0) * (k1 + 2.0 * k2 + 2.0 * k3 + k4)


def _ssprk53_step(f, y, t, dt):
    b10, b21, b32, b43, b54 = 0.377268915331368, 0.377268915331368, 0.242995220537396, 0.238458932846290, 0.287632146308408
    a30, a32, a40, a43, a52, a54 = (0.355909775063327, 0.644090224936674, 0.367933791638137, 0.632066208361863,
                                    0.237593836598569, 0.762406163401431)
    u1 = y + b10 * dt * f(y, t)
    u2 = u1 + b21 * dt * f(u1, t + 0.377268915331368 * dt)
    u3 = a30 * y + a32 * u2 + b32 * dt * f(u2, t + 0.754537830662736 * dt)
    u4 = a40 * y + a43 * u3 + b43 * dt * f(u3, t + 0.728985661612188 * dt)
    return a52 * u2 + a54 * u4 + b54 * dt * f(u4, t + 0.699226135931670 * dt)


def _envelope(t, t0, width, freq):
    x = t - t0
    return torch.exp(-(x / (2.0 * width)) ** 2) * torch.cos(freq * x)


def _cross(a, b):
    return torch.linalg.cross(a, b, dim=-1)


def _driven_rhs(m, t1, t2, a1, a2, width, freq):
    """dS/dt with the pulse pair of each trajectory ([B] tensors, or None), directions along (1,1,1) in the lab."""
    d = (m.frames @ _t([R3, R3, R3]))[None, None]

    def f(S, t):
        H = m.field(S)
        if a1 is not None:
            e = a1 * _envelope(t, t1, width, freq) + a2 * _envelope(t, t2, width, freq)
            H = H - e[:, None, None, None] * d
        return _cross(H, S)
    return f


def _fixed(m, f, y, T0, dt, steps, save, step=_rk4_step, want="rows"):
    """Rows (or states) every `save` steps and at the end, and the last state."""
    out, times, t = [], [], T0
    keep = m.rows if want == "rows" else (lambda s: s)
    for k in range(steps):
        if k % save == 0:
            out.append(keep(y))
            times.append(t)
        y = step(f, y, t, dt)
        t += dt
    return torch.stack(out + [keep(y)], 1), np.array(times + [t]), y


def exact(case, seed):
    x = _inputs(case, seed)
    kind = case["kind"]
    if kind == "uneven":
        return _exact_uneven(case, x)
    if kind == "mixed":
        return _exact_mixed(case, x)
    m = _model(case)
    shape = (-1, m.G, m.NA, 3)
    if kind == "adjoint":
        return _exact_adjoint(case, x, m, shape)
    if kind == "scan":
        B = case["B"]
        y = _t(x["states"]).reshape(shape).expand(B, -1, -1, -1)
        p = _t(x["pulses"]).T if case["drive"] else [None] * 4
        f = _driven_rhs(m, p[0], p[1], p[2], p[3], 0.5, 0.0)
        obs, _, y = _fixed(m, f, y, -5.0 if case["drive"] else 0.0, case["dt"], case["steps"], case["save"])
        return [obs, y.reshape(B, -1, 3)]
    y = _t(x["state"]).reshape(shape)
    amp, width, freq, t1, t2 = x["pulse"]
    one = lambda v, n=1: torch.full((n,), float(v), dtype=torch.float64, device=_DEV)
    if kind == "plain":
        f = _driven_rhs(m, one(t1), one(t2), one(amp) if case["drive"] else None, one(amp), width, freq)
        step = _rk4_step if case["method"] == "rk4" else _ssprk53_step
        ys, times, y = _fixed(m, f, y, 0.0, case["dt"], case["steps"], case["save"], step, "states")
        obs = torch.cat([m.rows(s) for s in ys[0].split(64)])
        return [obs, times, y.reshape(-1), [s.reshape(-1) for s in ys[0]] if case["states"] else []]
    B = case["B"]
    f = _driven_rhs(m, one(t1, B), _t(x["taus"]), one(amp, B), one(amp, B), width, freq)
    obs, times, _ = _fixed(m, f, y.expand(B, -1, -1, -1), -4.0, case["dt"], case["steps"], case["save"])
    return [times, obs[:, :, :9].transpose(0, 1).reshape(len(times), B, 3, 3)]


def _exact_adjoint(case, x, m, shape):
    """Loss, its derivative along each coupling (tangent of the discrete RK4 map), and M_local."""
    names = list(KITAEV) if case["lattice"] == "kitaev" else ["Jzz", "Jpm", "Jpmpm", "h"]
    basis = [_Model(case["lattice"], case["L1"], case["L2"], case["L3"], **{q: float(q == p) for q in names})
             for p in names]
    y = _t(x["states"]).reshape(shape)
    B, Q, n, target = case["B"], len(names), m.G * m.NA, _t(x["targets"])
    z = torch.zeros((Q,) + y.shape, dtype=torch.float64, device=_DEV)

    def f(u, t):
        S, dS = u[0], u[1:]
        H = m.field(S)
        dH = m.linear(dS.reshape(shape)).reshape(dS.shape) + torch.stack([b.field(S) for b in basis])
        return torch.cat([_cross(H, S)[None], _cross(dH, S.expand_as(dH)) + _cross(H.expand_as(dS), dS)])

    u, t = torch.cat([y[None], z]), 0.0
    loss, grad, mags = torch.zeros(B, dtype=torch.float64, device=_DEV), [], []
    grad = torch.zeros((Q, B), dtype=torch.float64, device=_DEV)
    for k in range(case["steps"] + 1):
        mag = u.sum((2, 3)) / n                              # [1 + Q, B, 3]
        r = mag[0] - target[:, k]
        loss, grad = loss + (r * r).sum(-1), grad + 2.0 * (r * mag[1:]).sum(-1)
        mags.append(mag[0])
        if k < case["steps"]:
            u = _rk4_step(f, u, t, case["dt"])
            t += case["dt"]
    return [loss, grad.T, torch.stack(mags, 1)]


# Dormand-Prince 5(4) (1980) and the step control of Boost.Odeint's controlled stepper.
_DP_A = [[1 / 5], [3 / 40, 9 / 40], [44 / 45, -56 / 15, 32 / 9], [19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729],
         [9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656],
         [35 / 384, 0.0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84]]
_DP_E = [35 / 384 - 5179 / 57600, 0.0, 500 / 1113 - 7571 / 16695, 125 / 192 - 393 / 640,
         -2187 / 6784 + 92097 / 339200, 11 / 84 - 187 / 2100, -1 / 40]


def _controlled(m, y, T1, dt0, tol, max_steps):
    """Rows {t, M..., E/N} after every accepted step of each trajectory (all capped by max_steps), and last states."""
    B = y.shape[0]
    t = torch.zeros(B, dtype=torch.float64, device=_DEV)
    dt = torch.full_like(t, dt0)
    done = torch.zeros(B, dtype=torch.long, device=_DEV)
    rows = torch.zeros((B, max_steps + 1, 11), dtype=torch.float64, device=_DEV)
    rows[:, 0, 1:] = m.rows(y)
    rhs = lambda s: _cross(m.field(s), s)
    ex = lambda v: v[:, None, None, None]
    k1, every = rhs(y), torch.arange(B, device=_DEV)
    while bool((done < max_steps).any()):
        dt = torch.where(t + dt > T1, T1 - t, dt)
        k = [k1]
        for row in _DP_A:
            u = y + ex(dt) * sum(a * kk for a, kk in zip(row, k) if a != 0.0)
            k.append(rhs(u))
        err = ex(dt) * sum(e * kk for e, kk in zip(_DP_E, k) if e != 0.0)
        e = (err.abs() / (tol + tol * (y.abs() + ex(dt) * k1.abs()))).amax((1, 2, 3))
        ok = (e <= 1.0) & (done < max_steps)
        t = torch.where(ok, t + dt, t)
        done = done + ok
        y, k1 = torch.where(ex(ok), u, y), torch.where(ex(ok), k[-1], k1)
        line = torch.cat([t[:, None], m.rows(y)], 1)
        rows[every[ok], done[ok]] = line[ok]
        grow = torch.where(e < 0.5, 0.9 * e.clamp(min=5.0 ** -5) ** -0.2, torch.ones_like(e))
        dt = dt * torch.where(e > 1.0, (0.9 * e ** (-1.0 / 3.0)).clamp(min=0.2), grow)
    return rows, y


def _exact_uneven(case, x):
    B = case["B"]
    rows, final = [None] * B, [None] * B
    for p in sorted(set(x["pick"].tolist())):
        at = [b for b in range(B) if x["pick"][b] == p]
        name, L = UNEVEN[p]
        m = _Model(name, L, L, 1 if name == "kitaev" else L, **_theta(name))
        y = _t(np.stack([x["states"][b] for b in at])).reshape(-1, m.G, m.NA, 3)
        r, y = _controlled(m, y, case["T1"], 0.01, case["tol"], case["max_steps"])
        for i, b in enumerate(at):
            rows[b], final[b] = r[i], y[i].reshape(-1)
    res = [torch.cat(rows), None]
    return res + [torch.cat(final)] if case["final"] else res


def _gell_mann_f():
    l = np.zeros((8, 3, 3), complex)
    for i, (a, b) in zip((0, 3, 5), ((0, 1), (0, 2), (1, 2))):
        l[i][a, b] = l[i][b, a] = 1
        l[i + 1][a, b], l[i + 1][b, a] = -1j, 1j
    l[2], l[7] = np.diag([1, -1, 0]), np.diag([1, 1, -2]) * R3
    f = np.einsum("aij,bjk,cki->abc", l, l, l)
    return (f - f.transpose(1, 0, 2)).imag / 4


def _exact_mixed(case, x):
    n, na = x["n"], x["na"]
    tab = {k: _t(x[k]).reshape((n,) + x[k].shape[2:]) for k in
           ("field2", "onsite2", "bil2", "part2", "mix2", "mp2", "field3", "onsite3", "bil3", "part3", "mix3", "mp3")}
    F, atom = _t(_gell_mann_f()), torch.arange(n, device=_DEV) % na
    drive = [_t(x["drive2"]), _t(x["drive3"])]

    def f(u, t):
        S = [u[: 3 * n].reshape(n, 3), u[3 * n:].reshape(n, 8)]
        H, t = [], torch.tensor(t, dtype=torch.float64, device=_DEV)
        e = [0.5 * _envelope(t, c, 0.5, 1.0) for c in (1.0, 2.0)]
        for i, s in enumerate("23"):
            h = 2.0 * torch.einsum("nij,nj->ni", tab["onsite" + s], S[i]) - tab["field" + s]
            h = h + torch.einsum("nzij,nzj->ni", tab["bil" + s], S[i][tab["part" + s]])
            h = h + torch.einsum("nzij,nzj->ni", tab["mix" + s], S[1 - i][tab["mp" + s]])
            H.append(h - e[0] * drive[i][0][atom] - e[1] * drive[i][1][atom])
        return torch.cat([_cross(H[0], S[0]).reshape(-1), torch.einsum("abc,nb,nc->na", F, H[1], S[1]).reshape(-1)])

    step = _rk4_step if case["method"] == "rk4" else _ssprk53_step
    ys, times, _ = _fixed(None, f, _t(x["state"])[None], 0.0, case["dt"], case["steps"], case["save"],
                          lambda g, y, t, dt: step(g, y[0], t, dt)[None], "states")
    return [times, list(ys[0])]
