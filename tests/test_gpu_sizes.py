"""The kernels that take any sizes, at the sizes where they can go wrong, against the general kernels
(SPO_B200_KERNELS=v1, which the oracle checks) or a numpy restatement (needs a B200).

  - kin_kernel: axis lengths and (x, y) grids without an instantiation, rectangular cells, odd basis sizes (lanes that
    do not pair up on 16-byte boundaries), one lane, the momentum shift;
  - potential5 (mixed) and potential4 (FP64) on the FP64 tensor cores: theta 1 to 16, phi 6 to 32, columns that do not
    fill an item or belong to several points, symmetry maps, the homonuclear basis;
  - the step as one graph against its kernels launched one by one;
  - host copies by several threads; prediction of the network for ragged numbers of points.

The bars are those of test_gpu_kernels.py: 1e-12 (FP64) and 2e-6 (mixed) of the largest value per operator, 1e-11 and 2e-5
relative L2 for an analysis step.
"""

import numpy as np
import pytest

from conftest import rel_err, rel_l2
from test_gpu_kernels import make

pytestmark = pytest.mark.gpu

TOL = {"fp64": (1e-12, 1e-11), "mixed": (2e-6, 2e-5)}


def random_state(case, seed):
    rng = np.random.default_rng(seed)
    psi = rng.standard_normal(case.psi_shape) + 1j * rng.standard_normal(case.psi_shape)
    return psi, rng.standard_normal(case.chi_shape) + 1j * rng.standard_normal(case.chi_shape)


def compare(case, precision, stages):
    """The default kernels against the general ones: the given operators one after another, then an analysis step."""
    psi, chi = random_state(case, 3)
    stage_bar, step_bar = TOL[precision]
    with make(case, "v1", precision) as ref, make(case, None, precision) as new:
        text = new.describe()
        for be in (ref, new):
            be.read_wave_packet(psi, chi)
        for stage in stages:
            for be in (ref, new):
                be.apply_stage(stage)
            a, b = ref.wave_packet_on_host(), new.wave_packet_on_host()
            assert rel_err(b[0], a[0]) < stage_bar and rel_err(b[1], a[1]) < stage_bar, (stage, text)
        for be in (ref, new):
            be.read_wave_packet(psi, chi)
            be.propagate_analysis_step()
        a, b = ref.wave_packet_on_host(), new.wave_packet_on_host()
        assert rel_l2(b[0], a[0]) < step_bar and rel_l2(b[1], a[1]) < step_bar, text
    return text


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nz,nr,nx,ny,j_max", [(90, 36, 10, 10, 2), (72, 45, 5, 9, 1), (110, 30, 9, 4, 2), (84, 44, 7, 7, 3),
                                               (60, 20, 16, 2, 1), (128, 48, 16, 16, 1), (176, 56, 4, 4, 2),
                                               (96, 40, 12, 12, 1), (36, 22, 3, 11, 0), (28, 18, 1, 1, 2),
                                               (192, 64, 6, 6, 1), (256, 48, 8, 8, 0), (224, 160, 2, 2, 1),
                                               (240, 14, 15, 14, 0)])
@pytest.mark.parametrize("shifted", [True, False])
def test_kinetic_passes_of_any_lengths(nz, nr, nx, ny, j_max, shifted, precision):
    from spo_b200 import capi, workload
    case = workload.config_case({"nz": nz, "nr": nr, "nx": nx, "ny": ny, "j_max": j_max, "mj_max": j_max,
                                 "nz_specular": 2 * nz, "nz_potential": nz // 3})
    if shifted:
        phase = np.exp(1j * np.random.default_rng(1).uniform(0, 6, nx * ny))
        case.a["shift_forward"], case.a["shift_backward"] = phase, np.conj(phase)
    compare(case, precision, (capi.STAGE_ZR, capi.STAGE_XY))


def fold(case, n):
    """C3v maps on an n x n cell: every point takes the potential of the smallest point of its orbit."""
    nphi, nt = case.n_phi, case.n_theta
    ix, iy = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    best, op, maps = np.full(n * n, n * n), np.zeros(n * n, dtype=np.int32), []
    for r in range(3):
        for s in (1, -1):
            x, y = (ix, iy) if s > 0 else (iy, ix)
            for _ in range(r):
                x, y = (-y) % n, (x - y) % n
            k = (x * n + y).ravel()
            op[k < best] = len(maps)
            best = np.minimum(best, k)
            maps.append((s * np.arange(nphi) + r * nphi // 3) % nphi)
    reps = np.unique(best)
    full = case.a["potential"].reshape(-1, n * n, nt * nphi)
    case.a["potential"] = np.ascontiguousarray(full[:, reps]).reshape(-1)
    case.a["representative_of"] = np.searchsorted(reps, best).astype(np.int32)
    case.a["operation_of"], case.a["phi_index"] = op, np.concatenate(maps).astype(np.int32)
    case.m["n_rep"], case.m["n_ops"] = len(reps), 6


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("j_max,homonuclear,nx,ny,symmetry",
                         [(j, False, 5, 3, False) for j in (2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 13, 14, 15)] +
                         [(4, True, 5, 3, False), (10, True, 4, 4, False), (14, True, 2, 2, False), (14, True, 8, 8, False),
                          (15, False, 2, 2, False), (15, False, 8, 8, False), (7, False, 1, 1, False),
                          (11, False, 6, 6, True), (8, False, 4, 4, True), (5, False, 3, 3, True)])
def test_potential_step_of_any_angular_grid(j_max, homonuclear, nx, ny, symmetry, precision):
    from spo_b200 import capi, workload
    case = workload.config_case({"nz": 16, "nr": 6, "nx": nx, "ny": ny, "j_max": j_max, "mj_max": j_max,
                                 "homonuclear": homonuclear, "nz_specular": 32, "nz_potential": 11})
    if symmetry:
        fold(case, nx)
    text = compare(case, precision, (capi.STAGE_POTENTIAL,))
    kernel = "potential4" if precision == "fp64" else "potential5"
    assert ",dmma" in text and f"potential={kernel}<nphi={case.n_phi}," in text, text


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("j_max,mj_max,homonuclear,nx,ny,symmetry",
                         [(13, 13, False, 4, 4, True), (15, 15, False, 4, 4, True), (12, 12, False, 6, 6, True),
                          (14, 13, False, 4, 4, True), (14, 13, False, 5, 3, False), (12, 12, False, 8, 8, False),
                          (15, 13, False, 5, 3, False), (13, 12, False, 2, 2, False), (9, 7, False, 5, 3, False),
                          (12, 7, False, 4, 4, True), (14, 11, True, 5, 3, False), (15, 2, False, 3, 3, False)])
def test_potential_step_where_lines_fill_the_registers_and_with_shorter_mj(j_max, mj_max, homonuclear, nx, ny, symmetry, precision):
    """potential5's ring (theta above 8, phi 28 and 32) with symmetry maps and with odd basis sizes (no bulk copies), and
    bases whose blocks are longer than phi asks for (mJ below J)."""
    from spo_b200 import capi, workload
    case = workload.config_case({"nz": 16, "nr": 6, "nx": nx, "ny": ny, "j_max": j_max, "mj_max": mj_max,
                                 "homonuclear": homonuclear, "nz_specular": 32, "nz_potential": 11})
    if symmetry:
        fold(case, nx)
    text = compare(case, precision, (capi.STAGE_POTENTIAL,))
    kernel = "potential4" if precision == "fp64" else "potential5"
    assert ",dmma" in text and f"potential={kernel}<nphi={case.n_phi}," in text, text


@pytest.mark.parametrize("nz,nr,nzs", [(6, 5, 6), (16, 16, 16), (16, 16, 33), (128, 64, 256), (128, 64, 512), (200, 90, 200)])
def test_sums_over_any_number_of_cells(nz, nr, nzs):
    """Averages and norm budget on grids of one block of cells, two, all 64 and more, twice each, one after the other (they share
    the count of blocks that have finished): the restatements' values to 1e-12, the second time to the last bit."""
    import norm_budget_oracle
    import spo_oracle
    from spo_b200 import workload
    case = workload.config_case({"nz": nz, "nr": nr, "nx": 1, "ny": 1, "j_max": 1, "mj_max": 1, "nz_specular": nzs,
                                 "nz_potential": 2})
    psi, chi = random_state(case, 4)
    for name, n in (("z_optical", nz), ("r_optical", nr), ("z_specular_optical", nzs)):
        case.a[name] = np.exp(-np.clip(np.linspace(-0.5, 0.2, n), 0.0, None))
    z, zs, r = 1.5 + 0.1 * np.arange(nz), 1.5 + 0.1 * np.arange(nzs), 0.4 + 0.1 * np.arange(nr)
    vols, line, surface = (0.02, 0.05), nz // 2, nzs - 2
    budget = norm_budget_oracle.NormBudgetOracle(case.a["z_optical"], case.a["r_optical"], case.a["z_specular_optical"],
                                                 case.steps_per_analysis, *vols, None, None)
    with make(case, None, "fp64") as be:
        be.norm_budget_setup(*vols)
        be.read_wave_packet(psi, chi)
        got = []
        for _ in range(3):
            got.append((be.averages(z, zs, r, *vols, line, surface), be.norm_budget_add()))
        dens = be.block_densities()
    want = spo_oracle.averages(dens, chi, z, zs, r, *vols, line, surface)
    assert np.max(np.abs(got[0][0] - want) / np.abs(want)) <= 1e-12
    budget.add(dens, chi)
    loss, err, start, end = budget.add(dens, chi)
    assert got[0][1] is None
    assert np.max(np.abs(got[1][1][0] - loss)) <= 1e-12 * end and np.max(np.abs(got[1][1][1] - err)) <= 1e-12 * end
    assert abs(got[1][1][2] - start) <= 1e-12 * end and abs(got[1][1][3] - end) <= 1e-12 * end
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[1][1][0], got[2][1][0]) and got[1][1][2:] == got[2][1][2:]


def uneven_blocks(sizes):
    """A case whose mJ blocks have the given lengths, m = -M .. M, and any matrices."""
    from spo_b200 import workload
    m_max = len(sizes) // 2
    case = workload.config_case({"nz": 16, "nr": 6, "nx": 5, "ny": 3, "j_max": m_max, "mj_max": m_max, "nz_specular": 32,
                                 "nz_potential": 11})
    rng = np.random.default_rng(sum(sizes))
    first = np.concatenate([[0], np.cumsum(sizes)[:-1]])
    case.m["n_rot"] = n_rot = sum(sizes)
    case.m["mj_blocks"] = [[int(f), n, b[2]] for f, n, b in zip(first, sizes, case.m["mj_blocks"])]
    case.m["initial_channel"] = int(first[m_max])
    case.a["legendre"] = rng.standard_normal(case.n_theta * n_rot) * 0.2
    case.a["rotation_half"] = np.exp(1j * rng.uniform(0, 6, n_rot * case.nr))
    return case


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("sizes,mma", [([1, 2, 3, 4, 3, 2, 1], True), ([2, 2, 3, 4, 3, 2, 1], True), ([1, 2, 3, 4, 3, 2, 5], True),
                                       ([13, 2, 3, 4, 3, 2, 1], False), ([4, 3, 2, 9, 9, 9, 30], True),
                                       ([30, 9, 9, 9, 2, 3, 4], False)])
def test_blocks_of_m_and_minus_m_may_differ_in_length(sizes, mma, precision):
    """The descriptor allows it. potential5 runs both with the steps of the longer one; where those would read more than the
    zeros behind a column, another kernel takes the grid."""
    from spo_b200 import capi
    text = compare(uneven_blocks(sizes), precision, (capi.STAGE_POTENTIAL,))
    if precision == "mixed":
        assert ("potential=potential5<" in text) == mma, text


@pytest.mark.parametrize("nz,nr", [(96, 24), (24, 96), (48, 24), (128, 24), (192, 24), (256, 24)])
def test_pairs_of_lanes_round_as_one_lane(nz, nr, monkeypatch):
    """Mixed form: where both kernels split a length the same way, a pair of lanes takes the same operations in the same order
    as a lane by itself, so kin_kernel's pass is as close to 64 bits as that of the kernel it replaces: equal but for a rare last
    bit (FMA contractions). 96 as 3 x 32 was not, 1e-7 apart."""
    from spo_b200 import capi, workload
    case = workload.config_case({"nz": nz, "nr": nr, "nx": 4, "ny": 4, "j_max": 5, "mj_max": 5, "nz_specular": 2 * nz,
                                 "nz_potential": nz // 3})
    psi, chi = random_state(case, 12)
    out = []
    for env in (None, "1"):
        if env:
            monkeypatch.setenv("SPO_B200_BALANCED", env)
        with make(case, None, "mixed") as be:
            axis = "z" if nz > 24 else "r"
            assert (f" {axis}=kin<{max(nz, nr)}=" in be.describe()) == (env is None), be.describe()
            be.read_wave_packet(psi, chi)
            be.apply_stage(capi.STAGE_ZR)
            out.append(be.wave_packet_on_host()[0])
    assert rel_l2(out[0], out[1]) < 2e-9, rel_l2(out[0], out[1])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_a_step_as_one_graph_is_bitwise_its_kernels_one_by_one(precision):
    """With profiling on the kernels are launched one after another on the handle's stream; the graph runs the specular
    grid's beside the kinetic passes. The same kernels on the same data, also on a caller's stream."""
    import torch
    from spo_b200 import workload
    case = workload.config_case({"nz": 48, "nr": 24, "nx": 6, "ny": 6, "j_max": 5, "mj_max": 5, "nz_specular": 96,
                                 "nz_potential": 30})
    psi, chi = random_state(case, 8)
    out = []
    for mode in ("graph", "launches", "stream"):
        with make(case, None, precision) as be:
            assert be.describe().endswith(" graph=1"), be.describe()
            be.read_wave_packet(psi, chi)
            if mode == "launches":
                be.profile(True)
            if mode == "stream":
                stream = torch.cuda.Stream()
                be.set_stream(stream.cuda_stream)
            for _ in range(3):
                be.propagate_analysis_step()
            out.append(be.wave_packet_on_host() + (be.last_launch_count(),))
    for other in out[1:]:
        assert np.array_equal(out[0][0], other[0]) and np.array_equal(out[0][1], other[1]) and out[0][2] == other[2]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_large_packets_cross_to_the_device_and_back_unchanged(precision):
    """Copies of 4 MiB and more by several threads: a packet that does not fill the last chunk, into ordinary and into
    pinned memory (which takes the other path)."""
    import torch
    from spo_b200 import workload
    case = workload.config_case({"nz": 64, "nr": 30, "nx": 7, "ny": 5, "j_max": 4, "mj_max": 4, "nz_specular": 128,
                                 "nz_potential": 4})
    psi, chi = random_state(case, 5)
    want = psi if precision == "fp64" else psi.astype(np.complex64).astype(np.complex128)
    with make(case, None, precision) as be:
        be.read_wave_packet(psi, chi)
        got, _ = be.wave_packet_on_host()
        assert np.array_equal(got, want)
        pinned = torch.empty(case.psi_shape, dtype=torch.complex128).pin_memory().numpy()
        pinned[...] = psi[::-1]
        be.read_wave_packet(pinned, None)
        got, _ = be.wave_packet_on_host()
        assert np.array_equal(got, want[::-1])


@pytest.mark.parametrize("n,n_in,width,depth", [(1, 1, 64, 1), (127, 12, 128, 2), (128, 64, 256, 4), (129, 7, 64, 8),
                                                (40001, 12, 256, 3), (200000, 12, 128, 4), (300001, 64, 64, 1)])
def test_predictions_of_ragged_numbers_of_points(n, n_in, width, depth):
    """Against the numpy oracle, to 1e-2 of the output scale (BF16 activations, as test_gpu_mlp.py)."""
    import mlp_oracle
    from spo_b200.mlp import Mlp
    x = np.random.default_rng(n).uniform(-1.0, 1.0, (n, n_in)).astype(np.float32)
    with Mlp(n_in, width, depth, seed=n) as net:
        some = np.unique(np.concatenate([np.arange(min(n, 300)), np.arange(max(0, n - 300), n)]))
        want, _, _ = mlp_oracle.forward(net.get_parameters(), x[some], net.input_width, width, depth)
        got = net.predict(x)
    assert got.shape == (n,) and np.all(np.isfinite(got))
    assert np.max(np.abs(got[some] - want)) <= 1e-2 * max(np.max(np.abs(want)), 1e-3)
