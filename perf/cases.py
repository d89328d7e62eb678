"""The calls whose speed this repository answers for: what a program that propagates wave packets on a
B200 has the library do, each through its public entry points.

A case is a dict of plain values. Its ``op`` says which calls a pass makes:

  step ......... one analysis step of the time loop: propagate, then the readbacks the loop makes after it
                 (the specular wave, the Z plane of the analysis line, the block densities)
  ensemble ..... the same for several uneven packets that advance by one graph launch
  restart ...... a packet handed in, one analysis step, the whole packet handed back (checkpoint)
  analysis ..... the device-side analysis of a resident packet: Balint-Kurti projection and S-matrix sums,
                 averages, norm budget
  predict ...... the learned potential on the points of a grid
  train ........ one epoch of its training, with the loss and the trained parameters

Sizes are those of the repository's configurations, tests and benchmark: the hard-wall configuration
(64 x 32 x 8 x 8, theta 8, phi 16), configuration 2/3 (128 x 48 x 16 x 16, theta 16, phi 32), the ensemble
ranges of configuration 4 (Z 96-128, r 40-48, x = y up to 12-16, theta 12-16, phi 24-32), the tiny test
cases (176 x 56 x 4 x 4, theta 4, phi 8) and lengths that no special kernel was made for.

``exact`` is a plain torch restatement in 64 bits (cuFFT and einsum over the whole arrays), independent of
the library's kernels and operator splitting.
"""

from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "cpp-spo-dvr_b200"))

from spo_b200 import B200Backend, Ensemble, workload  # noqa: E402
from spo_b200.mlp import Mlp  # noqa: E402

MIXED, FP64 = "mixed", "fp64"


def _grid(nz, nr, nx, ny, j, nzs, nzp, homo=False, sym=False):
    return dict(nz=nz, nr=nr, nx=nx, ny=ny, j=j, nzs=nzs, nzp=nzp, homo=homo, sym=sym)


# ------------------------------------------------------------------------------------------------
# The cases
# ------------------------------------------------------------------------------------------------
def listed():
    return [
        # The headline: configuration 3, one wave packet of 8.05e8 points in the mixed form.
        dict(name="step_config3_mixed", op="step", prec=MIXED, spa=5, **_grid(128, 48, 16, 16, 15, 512, 84)),
        # The FP64 form of the same set-up on a 12 x 12 cell, as a reference run of the mixed one is made.
        dict(name="step_fp64_12x12", op="step", prec=FP64, spa=5, **_grid(128, 48, 12, 12, 15, 512, 84)),
        # The hard-wall configuration (configuration 1): a small FP64 run of many steps.
        dict(name="step_hardwall_fp64", op="step", prec=FP64, spa=5, **_grid(64, 32, 8, 8, 7, 256, 42)),
        # A homonuclear molecule (H2: even J on the half theta grid), the reference's most common system.
        dict(name="step_h2_mixed", op="step", prec=MIXED, spa=5, **_grid(96, 40, 8, 8, 14, 320, 64, homo=True)),
        # The smallest runs (the repository's tiny test grids): launches and latency.
        dict(name="step_tiny_mixed", op="step", prec=MIXED, spa=5, **_grid(176, 56, 4, 4, 3, 280, 125)),
        # A user's own grid, of lengths that no register kernel is instantiated for.
        dict(name="step_ragged_mixed", op="step", prec=MIXED, spa=4, **_grid(90, 36, 10, 10, 8, 280, 55)),
        # A surface with C3v symmetry (UseSymmetry): the potential table folded by the point group.
        dict(name="step_c3v_mixed", op="step", prec=MIXED, spa=5, **_grid(96, 40, 12, 12, 11, 512, 64, sym=True)),
        # Configuration 4 on small cells: uneven packets advanced together, one of them in FP64.
        dict(name="ensemble_uneven", op="ensemble", members=6, pick=3, spa=5),
        # Restart and checkpoint of one packet around an analysis step.
        dict(name="restart_mixed", op="restart", prec=MIXED, spa=5, **_grid(64, 32, 8, 8, 7, 256, 42)),
        # The analysis after a step, on the device.
        dict(name="analysis_mixed", op="analysis", prec=MIXED, spa=5, **_grid(128, 48, 8, 8, 15, 512, 84)),
        # The learned potential (4 layers of 256) evaluated on a grid, and trained on one.
        dict(name="mlp_predict", op="predict", n=1000000, n_in=12, width=256, depth=4),
        dict(name="mlp_train", op="train", n=65536, batch=4096, n_in=12, width=256, depth=4),
    ]


_Z = [64, 72, 80, 84, 90, 96, 110, 112, 120, 128]
_R = [24, 30, 32, 36, 40, 44, 45, 48, 56]
_XY = [4, 5, 6, 8, 9, 10, 12]


def draw(rng):
    op = rng.choice(["step"] * 8 + ["ensemble", "restart", "analysis", "predict", "train"])
    if op in ("predict", "train"):
        width = rng.choice([64, 128, 256, 256])
        depth = rng.choice([2, 3, 4, 4, 5])
        n_in = rng.randint(6, 24)
        if op == "predict":
            return dict(op=op, n=int(10 ** rng.uniform(3.5, 6.0)), n_in=n_in, width=width, depth=depth)
        batch = rng.choice([1024, 2048, 4096, 8192])
        return dict(op=op, n=batch * rng.randint(2, 8) + rng.randint(0, batch - 1), batch=batch, n_in=n_in, width=width,
                    depth=depth)
    if op == "ensemble":
        return dict(op=op, members=rng.randint(2, 6), pick=rng.randint(4, 10 ** 6), spa=rng.choice([2, 4, 5]))
    nz, nr = rng.choice(_Z), rng.choice(_R)
    nx = rng.choice(_XY)
    ny = nx if rng.random() < 0.75 else rng.choice(_XY)
    homo = rng.random() < 0.3
    j = rng.choice([4, 6, 8, 10, 12, 14] if homo else [3, 5, 6, 7, 9, 11, 12, 13, 15])
    sym = nx == ny and not homo and j == 11 and rng.random() < 0.7
    while nz * nr * nx * ny * (j + 1) ** 2 > 1.2e8:
        nx = ny = max(4, nx - 2)
        if nx == 4 and nz * nr * nx * ny * (j + 1) ** 2 > 1.2e8:
            nz = 64
            break
    return dict(op=op, prec=rng.choice([MIXED, MIXED, FP64]), spa=rng.choice([2, 4, 5]),
                **_grid(nz, nr, nx, ny, j, nz * rng.choice([2, 4]), int(nz * rng.uniform(0.5, 0.68)), homo, sym))


def _members(case):
    """Members of an ensemble: grids of configuration 4's Z, r and angular ranges on small cells. Its sizes
    are made from `pick` alone."""
    rng = np.random.default_rng(case["pick"])
    out = []
    for k in range(case["members"]):
        nxy = int(rng.choice([4, 6, 8]))
        out.append(dict(prec=FP64 if k == 1 else MIXED, spa=case["spa"],
                        **_grid(int(rng.choice([96, 112, 128])), int(rng.choice([40, 48])), nxy, nxy,
                                int(rng.choice([7, 11, 13, 15])), 512, int(rng.choice([60, 70])))))
    return out


# ------------------------------------------------------------------------------------------------
# Inputs
# ------------------------------------------------------------------------------------------------
def _fft_size(n):
    """Whether the library transforms length n (2^h 3^i 5^j 7^k 11^m)."""
    for p in (2, 3, 5, 7, 11):
        while n % p == 0:
            n //= p
    return n == 1


def _symmetry(n, n_phi):
    """C3v on an n x n hexagonal cell: representatives, operations and phi maps. Operation (r, s) takes phi to
    s phi + r n_phi / 3 on the phi grid; every point takes V of the smallest point of its orbit."""
    ix, iy = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    best, op = np.full(n * n, n * n), np.zeros(n * n, dtype=np.int32)
    phi = np.arange(n_phi)
    maps = []
    for r in range(3):
        for s in (1, -1):
            x, y = (ix, iy) if s > 0 else (iy, ix)
            for _ in range(r):
                x, y = (-y) % n, (x - y) % n
            k = (x * n + y).ravel()
            better = k < best
            best[better] = k[better]
            op[better] = len(maps)
            maps.append((s * phi + r * n_phi // 3) % n_phi)
    reps = np.unique(best)
    return reps, np.searchsorted(reps, best).astype(np.int32), op, np.concatenate(maps).astype(np.int32)


def _bundle(c, seed):
    """The case bundle of a grid: the tables of a wave packet on it, with a corrugation, an incident packet and
    a shape of V of their own for each seed."""
    rng = np.random.default_rng(seed)
    case = workload.config_case(dict(nz=c["nz"], nr=c["nr"], nx=c["nx"], ny=c["ny"], j_max=c["j"], mj_max=c["j"],
                                     homonuclear=c["homo"], nz_specular=c["nzs"], nz_potential=1,
                                     steps_per_analysis=c["spa"]))
    m, a = case.m, case.a
    nx, ny, nr, nzp, nt, nphi = c["nx"], c["ny"], c["nr"], c["nzp"], m["n_theta"], m["n_phi"]
    reps = np.arange(nx * ny)
    if c["sym"]:
        reps, a["representative_of"], a["operation_of"], a["phi_index"] = _symmetry(nx, nphi)
        m["n_rep"], m["n_ops"] = len(reps), 6
    # V = A(Z, r) + B(Z) g(x, y, theta, phi), capped at 0.5 hartree
    z = 0.12 * np.arange(nzp) * (128.0 / c["nz"])
    r = 0.5 + 0.16 * np.arange(nr)
    u, v = reps // ny / nx, reps % ny / ny
    amp = rng.uniform(0.06, 0.12, 3)
    corr = amp[0] * np.cos(2 * np.pi * u) + amp[1] * np.cos(2 * np.pi * v) + amp[2] * np.cos(2 * np.pi * (u - v))
    cos_t = np.linspace(0.95, 0.05 if c["homo"] else -0.95, nt)
    phi = 2 * np.pi * np.arange(nphi) / nphi
    ang = 1 + rng.uniform(0.2, 0.4) * (1 - cos_t ** 2)[:, None] * np.cos(2 * phi + rng.uniform(0, 6))[None, :]
    g = torch.from_numpy(((0.5 + corr)[:, None, None] * ang[None]).reshape(1, -1))
    vasy = 0.1745 * (1 - np.exp(-1.02 * (r - 1.4))) ** 2
    A = 0.07 * (np.exp(-2.2 * (z - 2.5)) - 2 * np.exp(-1.1 * (z - 2.5)))[:, None] + vasy[None, :]
    B = 0.05 * np.exp(-0.8 * (z - 1.5)).clip(max=10.0)[:, None] * np.ones((1, nr))
    pot = torch.empty((nzp, nr, g.numel()), dtype=torch.float64)
    for iz in range(nzp):
        torch.addcmul(torch.from_numpy(A[iz])[:, None], torch.from_numpy(B[iz])[:, None], g, out=pot[iz])
        pot[iz].clamp_(max=0.5)
    a["potential"] = pot.numpy().reshape(-1)
    m["nz_potential"] = nzp
    zs = np.arange(c["nzs"]) / c["nzs"]
    packet = np.exp(-200 * (zs - rng.uniform(0.3, 0.5)) ** 2 - 1j * rng.uniform(60, 90) * zs)
    chi_r = np.exp(-8.0 * (r - 1.4) ** 2)
    a["chi_initial"] = (packet[:, None] * chi_r[None, :]).ravel().astype(np.complex128)
    return case


def _packet(case, seed):
    """A wave packet in mid run, on the host: two Gaussians in (Z, r), each with its own momentum and its own
    amplitudes on the (x, y) points and the rotational states."""
    rng = np.random.default_rng(seed + 7)
    z, r = np.arange(case.nz) / case.nz, np.arange(case.nr) / case.nr
    left = []
    for _ in range(2):
        gz = np.exp(-12 * (z - rng.uniform(0.3, 0.7)) ** 2 + 1j * rng.uniform(-60, 60) * z)
        gr = np.exp(-12 * (r - rng.uniform(0.3, 0.7)) ** 2 + 1j * rng.uniform(-30, 30) * r)
        left.append((gz[:, None] * gr[None, :]).ravel())
    n = case.nx * case.ny * case.n_rot
    j = np.tile(np.asarray(case.j, dtype=np.float64), case.nx * case.ny)
    right = (rng.standard_normal((2, n)) + 1j * rng.standard_normal((2, n))) * np.exp(-j / 8.0) * 1e-2
    return torch.from_numpy(np.stack(left, axis=1)) @ torch.from_numpy(right)  # (nz nr, nx ny n_rot)


def _pinned(shape):
    t = torch.empty(shape, dtype=torch.complex128)
    return (t.pin_memory() if torch.cuda.is_available() else t).numpy()


def _backend(c, seed):
    case = _bundle(c, seed)
    be = B200Backend(case, precision=c["prec"])
    be.read_wave_packet(_packet(case, seed).numpy(), case.a["chi_initial"])
    # what the handle was built from is on the device now; the program keeps the sizes
    return be, _pinned(case.chi_shape), _pinned((case.nr, case.nx, case.ny, case.n_rot))


def _mlp_inputs(case, seed):
    g = torch.Generator().manual_seed(seed)
    x = torch.rand((case["n"], case["n_in"]), generator=g) * 2 - 1
    w = torch.randn((case["n_in"],), generator=g)
    y = torch.sin(x @ w) * 0.3 + 0.2 * x[:, 0] * x[:, -1]
    return x.numpy(), y.numpy().astype(np.float32)


def _mlp_parameters(case, seed):
    """Weights as a trained or freshly initialised network has them (uniform, scaled by the fan-in)."""
    rng = np.random.default_rng(seed + 1)
    out = []
    for layer in range(case["depth"]):
        fan = case["n_in"] if layer == 0 else case["width"]
        cols = 64 if layer == 0 else case["width"]
        w = rng.uniform(-1, 1, (case["width"], cols)) * math.sqrt(3.0 / fan)
        w[:, fan:] = 0.0
        out += [w.ravel(), rng.uniform(-0.1, 0.1, case["width"])]
    out += [rng.uniform(-1, 1, case["width"]) * math.sqrt(3.0 / case["width"]), rng.uniform(-0.1, 0.1, 1)]
    return np.concatenate(out).astype(np.float32)


def _analysis_tables(case, seed):
    rng = np.random.default_rng(seed + 3)
    n_v, j_max = 3, max(case.j)
    rot = [k for k, j in enumerate(case.j) if j <= 7]
    nx, ny = case.nx, case.ny
    half = [(ix, iy) for ix in (0, 1, 2, nx - 1, nx - 2) for iy in (0, 1, ny - 1)]
    r = np.linspace(-3, 3, case.nr)
    phi = np.empty((n_v, j_max + 1, case.nr))
    for v in range(n_v):
        for j in range(j_max + 1):
            phi[v, j] = np.exp(-r ** 2) * (1 + rng.uniform(0.5, 1.5) * r) ** v
    energies = np.linspace(0.2, 1.0, 41) / 27.2114 + 0.01
    a = dict(n_v=n_v, n_rotation=len(rot), n_diffraction=len(half), rotation_index=rot,
             rotation_j=[case.j[k] for k in rot], channel_ix=[h[0] for h in half], channel_iy=[h[1] for h in half],
             j_max_gas=j_max, initial_state=0, j_in=0, iz_analysis=case.iz_analysis, dr=case.dr, xy_scale=0.3,
             analysis_time_step=2.0 * case.steps_per_analysis)
    grids = (0.12 * np.arange(case.nz), 0.12 * np.arange(case.nz_specular), 0.5 + 0.16 * np.arange(case.nr))
    return a, phi.ravel(), energies, grids


_VOLUMES = (0.12 * 0.16 * 0.37, 0.12 * 0.16)


def prepare(case, seed):
    op = case["op"]
    if op in ("step", "restart", "analysis"):
        be, chi, plane = _backend(case, seed)
        s = dict(op=op, be=be, chi=chi, plane=plane, iz=be.case.iz_analysis)
        if op == "restart":
            s["psi0"], s["chi0"] = _packet(be.case, seed).numpy().copy(), be.case.a["chi_initial"].copy()
        if op == "analysis":
            a, phi, energies, grids = _analysis_tables(be.case, seed)
            be.analysis_setup(a, phi, energies)
            be.norm_budget_setup(*_VOLUMES)
            be.norm_budget_add()
            s.update(grids=grids, t=0.0, dt=a["analysis_time_step"], surface=int(0.9 * be.case.nz))
        be.case.a = {}
        return s
    if op == "ensemble":
        made = [_backend(c, seed + 100 * k) for k, c in enumerate(_members(case))]
        for be, _, _ in made:
            be.case.a = {}
        return dict(op=op, made=made, ens=Ensemble([m[0] for m in made]))
    x, y = _mlp_inputs(case, seed)
    net = Mlp(case["n_in"], case["width"], case["depth"], seed=1)
    net.set_parameters(_mlp_parameters(case, seed))
    return dict(op=op, net=net, x=x, y=y, batch=case.get("batch", 0), seed=seed)


# ------------------------------------------------------------------------------------------------
# The passes
# ------------------------------------------------------------------------------------------------
def run(s):
    op = s["op"]
    if op == "step":
        be = s["be"]
        be.propagate_analysis_step()
        return [be.specular(out=s["chi"]), be.z_plane(s["iz"], out=s["plane"]), be.block_densities()]
    if op == "ensemble":
        s["ens"].propagate_analysis_step()
        return [[be.specular(out=chi), be.z_plane(be.case.iz_analysis, out=plane)] for be, chi, plane in s["made"]]
    if op == "restart":
        be = s["be"]
        be.read_wave_packet(s["psi0"], s["chi0"])
        be.propagate_analysis_step()
        return list(be.wave_packet_on_host())
    if op == "analysis":
        be, (z, zs, r) = s["be"], s["grids"]
        s["t"] += s["dt"]
        bk = be.bk_coefficients(s["t"], accumulate=True)
        av = be.averages(z, zs, r, *_VOLUMES, s["iz"], s["surface"])
        loss, err, start, end = be.norm_budget_add()
        return [bk, be.s_matrix_sums(), av, loss, err, start, end]
    if op == "predict":
        return [s["net"].predict(s["x"])]
    loss = s["net"].train(s["x"], s["y"], epochs=1, batch=s["batch"], lr=1e-3, seed=s["seed"])
    return [loss, s["net"].get_parameters()]


# ------------------------------------------------------------------------------------------------
# What a pass cannot do without
# ------------------------------------------------------------------------------------------------
def _angles(c):
    """(n_rot, theta, phi) of a grid with JMax = MJMax = j."""
    j, step = c["j"], 2 if c["homo"] else 1
    n_rot = sum(len([k for k in range(0, j + 1, step) if k >= abs(m)]) for m in range(-j, j + 1))
    n_phi = 2 * j + 1
    while n_phi % 2 or not _fft_size(n_phi):
        n_phi += 1
    return n_rot, (j + 2) // 2 if c["homo"] else j + 1, n_phi


def _step_work(c):
    """One analysis step: per time step psi moves once for T and once for V (interaction region only), and the
    table exp(-iV dt) and the specular wave once; the transforms and the two theta contractions."""
    s = 16.0 if c["prec"] == FP64 else 8.0
    n_rot, nt, nphi = _angles(c)
    lanes, nxy, part = c["nx"] * c["ny"] * n_rot, c["nx"] * c["ny"], c["nzp"] / c["nz"]
    n_psi, n_chi = c["nz"] * c["nr"] * lanes, c["nzs"] * c["nr"]
    n_rep = len(_symmetry(c["nx"], nphi)[0]) if c["sym"] else nxy
    n_tab = c["nzp"] * c["nr"] * n_rep * nt * nphi
    per = s * (2 * n_psi + 2 * part * n_psi + n_tab + 4 * n_chi)
    fft = 10.0 * n_psi * math.log2(c["nz"] * c["nr"] * nxy) + 6.0 * 3 * n_psi
    dvr = c["nzp"] * c["nr"] * nxy * nt * nphi
    pot = 2 * 4.0 * nt * n_psi * part + 10.0 * dvr * math.log2(nphi) + 6.0 * dvr
    plane = 16.0 * (c["nr"] * lanes + n_chi)
    return {"bytes": c["spa"] * per + plane, "flops": c["spa"] * (fft + pot)}


def work(case):
    op = case["op"]
    if op == "step":
        return _step_work(case)
    if op == "ensemble":
        w = [_step_work(c) for c in _members(case)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    if op == "restart":
        w = _step_work(case)
        n = case["nz"] * case["nr"] * case["nx"] * case["ny"] * _angles(case)[0] + case["nzs"] * case["nr"]
        return {"bytes": w["bytes"] + 2 * n * (16.0 + (16.0 if case["prec"] == FP64 else 8.0)), "flops": w["flops"]}
    if op == "analysis":
        n_rot, _, _ = _angles(case)
        n = case["nz"] * case["nr"] * case["nx"] * case["ny"] * n_rot
        states = len([1 for m in range(-7, 8) for j in range(8) if j >= abs(m)]) * 15 * 3
        return {"bytes": (16.0 if case["prec"] == FP64 else 8.0) * n + 3 * 16.0 * states * 41, "flops": 4.0 * n + 8.0 * states * 41}
    weights = 64 * case["width"] + (case["depth"] - 1) * case["width"] ** 2
    if op == "predict":
        return {"bytes": 4.0 * case["n"] * (case["n_in"] + 1) + 2.0 * weights, "flops": 2.0 * case["n"] * weights}
    steps = case["n"] // case["batch"]
    return {"bytes": 4.0 * case["n"] * (case["n_in"] + 1) + steps * 24.0 * weights,
            "flops": 6.0 * steps * case["batch"] * weights}


def tolerance(case):
    """Measured against ``exact`` and stated about four times larger, with room for three passes on one state:
    FP64 packets differ by 3e-15 after a step, complex64 packets by 3e-7 to 6e-7, the bf16 network by 3e-3
    (predictions) and 8e-4 after an epoch (parameters, whose Adam updates follow the signs of small gradients, so
    that the difference grows by as much with every further epoch)."""
    op = case["op"]
    if op == "predict":
        return {"rel": 1.2e-2, "max": 0.1}
    if op == "train":
        return {"rel": 1e-2, "max": 0.4}
    if op == "ensemble" or case["prec"] == MIXED:
        return {"rel": 2.4e-6, "max": 3e-4}
    return {"rel": 2e-14, "max": 2e-12}


# ------------------------------------------------------------------------------------------------
# The same in 64 bits, by plain torch
# ------------------------------------------------------------------------------------------------
def _propagate(case, psi, chi):
    """One analysis step in complex128 on the GPU: psi (nz, nr, nx, ny, n_rot), chi (nz_specular, nr)."""
    m, dev = case, psi.device
    t = {k: torch.from_numpy(np.ascontiguousarray(v)).to(dev) for k, v in case.a.items() if k != "potential"}
    nz, nr, nx, ny, n_rot, nzp, nt, nphi = m.nz, m.nr, m.nx, m.ny, m.n_rot, m.nz_potential, m.n_theta, m.n_phi
    rot = t["rotation_half"].reshape(nr, n_rot)
    gas = rot * t["gas_phase"][:, None] * rot
    i0, first, last = m.initial_channel, m.r_absorber_first, m.r_absorber_last
    opt_r, opt_z = t["r_optical"], t["z_optical"]
    mats, off = [], 0
    for f, n, slot in np.asarray(m.mj_blocks).reshape(-1, 3):
        mats.append((int(f), int(n), int(slot), t["legendre"][off:off + nt * n].reshape(nt, n).to(torch.complex128)))
        off += nt * n
    rep, op, maps = t["representative_of"].long(), t["operation_of"].long(), t["phi_index"].long().reshape(-1, nphi)
    sc2sp, sp2sc = t["scattering_to_specular"], t["specular_to_scattering"]
    folded = m.n_rep < nx * ny
    V = torch.from_numpy(case.a["potential"]).reshape(nzp, nr, m.n_rep, nt, nphi)
    n = m.steps_per_analysis
    for k in range(n + 1):
        f = "half" if k in (0, n) else "full"
        x = torch.fft.ifft2(torch.fft.fft2(chi) * t["specular_kinetic_" + f].reshape(m.nz_specular, nr))
        if k < n:
            x[nzp:] *= gas[None, :, i0]
            x *= t["z_specular_optical"][:, None]
            x[:, first:last + 1] *= opt_r[None, first:last + 1]
        chi = x
        for dim, name in ((0, "z"), (1, "r")):
            shape = [1] * 5
            shape[dim] = -1
            for q in range(0, nx):  # by x: bounded temporary memory
                part = torch.fft.fft(psi[:, :, q], dim=dim)
                part *= t[name + "_kinetic_" + f].reshape(shape[:4])
                psi[:, :, q] = torch.fft.ifft(part, dim=dim)
        xy = t["xy_kinetic_" + f].reshape(nx, ny, 1)
        for iz in range(nz):
            p = torch.fft.ifft2(torch.fft.fft2(psi[iz], dim=(1, 2)) * xy, dim=(1, 2))
            if k < n and iz >= nzp:
                p = p * (opt_z[iz] * opt_r[:, None] * gas)[:, None, None, :]
            psi[iz] = p
        if k == n:
            break
        for iz in range(nzp):
            p = psi[iz].reshape(nr, nx * ny, n_rot) * (opt_z[iz] * opt_r[:, None] * rot)[:, None, :]
            p[:, :, i0] += rot[:, i0][:, None] * sp2sc[None, :] * chi[iz][:, None]
            d = torch.zeros((nr, nx * ny, nt, nphi), dtype=torch.complex128, device=dev)
            for a, cnt, slot, mat in mats:
                d[..., slot] = p[..., a:a + cnt] @ mat.T
            e = V[iz].to(dev)
            if folded:
                e = e[:, rep].gather(3, maps[op][None, :, None, :].expand(nr, -1, nt, -1))
            d = torch.fft.ifft(d, dim=3, norm="forward") * torch.polar(torch.ones_like(e), e * -m.time_step)
            d = torch.fft.fft(d, dim=3)
            for a, cnt, slot, mat in mats:
                p[..., a:a + cnt] = d[..., slot] @ mat
            p *= rot[:, None, :]
            chi[iz] = p[:, :, i0] @ sc2sp
            p[:, :, i0] -= sp2sc[None, :] * chi[iz][:, None]
            psi[iz] = p.reshape(nr, nx, ny, n_rot)
    return psi, chi


def _exact_state(c, seed):
    case = _bundle(c, seed)
    psi = _packet(case, seed).reshape(case.psi_shape).cuda()
    return case, psi, torch.from_numpy(case.a["chi_initial"]).reshape(case.chi_shape).cuda()


def _densities(psi):
    return torch.stack([p.abs().square().sum(dim=(1, 2, 3)) for p in psi]).reshape(-1)


def _exact_analysis(c, seed):
    case, psi, chi = _exact_state(c, seed)
    a, phi, energies, (z, zs, r) = _analysis_tables(case, seed)
    phi = torch.from_numpy(phi).reshape(a["n_v"], -1, case.nr).cuda()
    plane = psi[case.iz_analysis]  # (nr, nx, ny, n_rot)
    bk = torch.empty((a["n_v"], a["n_rotation"], a["n_diffraction"]), dtype=torch.complex128, device="cuda")
    ix, iy = torch.tensor(a["channel_ix"]), torch.tensor(a["channel_iy"])
    for i, (k, j) in enumerate(zip(a["rotation_index"], a["rotation_j"])):
        o = torch.einsum("rxy,vr->vxy", plane[..., k], phi[:, j].to(torch.complex128)) * a["dr"]
        bk[:, i] = torch.fft.fft2(o)[:, ix.cuda(), iy.cuda()] * a["xy_scale"]
    bk = bk.reshape(-1)
    t1 = a["analysis_time_step"]
    sums = torch.polar(torch.ones(len(energies), dtype=torch.float64), torch.from_numpy(energies) * t1).cuda()[:, None] * bk[None] * t1
    d, ds = _densities(psi).reshape(case.nz, case.nr), chi.abs().square()
    gz, gzs, gr = (torch.from_numpy(g).cuda() for g in (z, zs, r))
    v0, v1 = _VOLUMES
    norm = d.sum() * v0 + ds.sum() * v1
    iz, surface = case.iz_analysis, int(0.9 * case.nz)
    av = [norm, ((d * gz[:, None]).sum() * v0 + (ds * gzs[:, None]).sum() * v1) / norm,
          ((d * gr[None]).sum() * v0 + (ds * gr[None]).sum() * v1) / norm, ds[iz + 1:surface + 1].sum() * v1]
    # the packet has not moved since the budget's window began
    loss, err = [], []
    vr = -torch.log(torch.from_numpy(case.a["r_optical"]).cuda())[None, :]
    for rho, f in ((d * v0, case.a["z_optical"]), (ds * v1, case.a["z_specular_optical"])):
        vz = -torch.log(torch.from_numpy(f).cuda())[:, None]
        g = 2 * c["spa"] * (vz + vr)
        cell = torch.where(g > 0, rho * -torch.expm1(-g) + rho * -torch.expm1(-g) * (g / -torch.expm1(-g) - 1), torch.zeros_like(g))
        cell = torch.where(g > 0, cell, torch.zeros_like(cell))
        e = g * g / 6 * cell.abs()
        share = torch.where(g > 0, vz / (vz + vr).clamp(min=1e-300), torch.zeros_like(g))
        loss += [(share * cell).sum(), ((1 - share) * cell).sum()]
        err += [(share * e).sum(), ((1 - share) * e).sum()]
    total = float(norm)
    return [bk.cpu().numpy(), sums.cpu().numpy(), torch.stack(av).cpu().numpy(), torch.stack(loss).cpu().numpy(),
            torch.stack(err).cpu().numpy(), total, total]


def _network(case, p):
    """Weights and biases of a parameter vector, in 64 bits on the GPU."""
    p, out, off = torch.from_numpy(p).double().cuda(), [], 0
    for layer in range(case["depth"]):
        cols = 64 if layer == 0 else case["width"]
        out += [p[off:off + case["width"] * cols].reshape(case["width"], cols)]
        off += case["width"] * cols
        out += [p[off:off + case["width"]]]
        off += case["width"]
    return out + [p[off:off + case["width"]], p[off + case["width"]:]]


def _forward(case, net, x):
    h = torch.nn.functional.pad(x, (0, 64 - case["n_in"]))
    for layer in range(case["depth"]):
        h = torch.nn.functional.silu(h @ net[2 * layer].T + net[2 * layer + 1])
    return h @ net[-2] + net[-1]


def _batch_order(n, seed):
    """The library's order of an epoch's points: a Fisher-Yates shuffle driven by splitmix64."""
    mask, s, order = (1 << 64) - 1, seed, list(range(n))
    for i in range(n - 1, 0, -1):
        s = (s + 0x9E3779B97F4A7C15) & mask
        z = ((s ^ (s >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        k = (z ^ (z >> 31)) % (i + 1)
        order[i], order[k] = order[k], order[i]
    return order


def _exact_train(case, seed):
    x, y = (torch.from_numpy(v).double().cuda() for v in _mlp_inputs(case, seed))
    net = [p.clone().requires_grad_() for p in _network(case, _mlp_parameters(case, seed))]
    first, second = [torch.zeros_like(p) for p in net], [torch.zeros_like(p) for p in net]
    order = torch.tensor(_batch_order(case["n"], seed)).cuda()
    steps, total = case["n"] // case["batch"], 0.0
    for t in range(steps):
        rate = 1e-3 * (0.05 + 0.95 * 0.5 * (1 + math.cos(math.pi * t / max(steps - 1, 1))))
        at = order[t * case["batch"]:(t + 1) * case["batch"]]
        loss = (_forward(case, net, x[at]) - y[at]).square().mean()
        total += float(loss)
        with torch.no_grad():
            for p, m, v, g in zip(net, first, second, torch.autograd.grad(loss, net)):
                m.mul_(0.9).add_(g, alpha=0.1)
                v.mul_(0.999).add_(g * g, alpha=0.001)
                p -= rate * (m / (1 - 0.9 ** (t + 1))) / ((v / (1 - 0.999 ** (t + 1))).sqrt() + 1e-8)
    return [total / steps, torch.cat([p.detach().reshape(-1) for p in net]).float().cpu().numpy()]


def exact(case, seed):
    op = case["op"]
    if op in ("step", "restart"):
        c, psi, chi = _exact_state(case, seed)
        psi, chi = _propagate(c, psi, chi)
        if op == "restart":
            return [psi.cpu().numpy(), chi.cpu().numpy()]
        return [chi.cpu().numpy(), psi[c.iz_analysis].cpu().numpy(), _densities(psi).cpu().numpy()]
    if op == "ensemble":
        out = []
        for k, member in enumerate(_members(case)):
            c, psi, chi = _exact_state(member, seed + 100 * k)
            psi, chi = _propagate(c, psi, chi)
            out.append([chi.cpu().numpy(), psi[c.iz_analysis].cpu().numpy()])
        return out
    if op == "analysis":
        return _exact_analysis(case, seed)
    if op == "predict":
        x = torch.from_numpy(_mlp_inputs(case, seed)[0])
        net = _network(case, _mlp_parameters(case, seed))
        return [torch.cat([_forward(case, net, p.double().cuda()) for p in x.split(1 << 17)]).cpu().numpy()]
    return _exact_train(case, seed)
