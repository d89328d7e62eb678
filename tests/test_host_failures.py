"""The library's host code where calls of the CUDA runtime fail, and what it leaves behind (CPU only).

tests/support/fake_cudart.cpp stands in for the runtime: device memory is host memory, kernels are not run, every object
is counted, and a chosen call can be made to fail. Each check runs in a process of its own with that library preloaded.
"""

import os
import subprocess
import sys

import pytest

from conftest import ROOT

PKG = os.path.join(ROOT, "cpp-spo-dvr_b200")
PRELUDE = """
import ctypes, os, sys
import numpy as np
sys.path.insert(0, %r)
from spo_b200 import B200Backend, Ensemble, capi, workload
from spo_b200.mlp import Mlp
fake = ctypes.CDLL(None)
fake.fake_launches.restype = ctypes.c_long
fake.fake_bytes.restype = ctypes.c_longlong
KINDS = (b"malloc", b"host", b"stream", b"event", b"graph", b"exec")
live = lambda: {k.decode(): fake.fake_live(k) for k in KINDS if fake.fake_live(k)}
def status(call):
    try:
        call()
        return capi.SPO_OK
    except capi.B200Error as e:
        return e.status
def case(nz=24, nr=12, nx=4, ny=4, j=3, nzp=10, **kw):
    return workload.config_case({"nz": nz, "nr": nr, "nx": nx, "ny": ny, "j_max": j, "mj_max": j, "nz_specular": 2 * nz,
                                 "nz_potential": nzp, **kw})
""" % PKG


@pytest.fixture(scope="session")
def run(tmp_path_factory):
    """run(code): the code after PRELUDE, with the stand-in preloaded; fails with its output unless it ends well."""
    lib = os.path.join(PKG, "lib", "libspo_b200.so")
    if not os.path.exists(lib):
        subprocess.run(["make", "-C", PKG, "-j4"], check=True, stdout=subprocess.DEVNULL)
    fake = str(tmp_path_factory.mktemp("fake") / "libfake_cudart.so")
    include = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", f"-I{include}", "-o", fake,
                    os.path.join(ROOT, "tests", "support", "fake_cudart.cpp")], check=True)

    def go(code, env=None):
        r = subprocess.run([sys.executable, "-c", PRELUDE + code], env={**os.environ, "LD_PRELOAD": fake, **(env or {})},
                           capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr

    return go


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_a_handle_asks_for_no_pinned_memory(run, precision):
    """Page-locked memory takes milliseconds to get and to give back; a handle that copies nothing large needs none."""
    run(f"""
with B200Backend(case(), precision="{precision}") as be:
    be.propagate_analysis_step()
    be.block_densities()
assert fake.fake_calls(b"host") == 0
""")


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("kind", ["malloc", "stream", "event"])
def test_a_handle_that_cannot_be_made_leaves_nothing_behind(run, kind, precision):
    """Every call of a kind that making a handle needs, failing once: the status says so and nothing stays alive."""
    run(f"""
c = case()
B200Backend(c, precision="{precision}").close()
n = fake.fake_calls(b"{kind}")
assert n > 0 and not live(), (n, live())
for k in range(1, n + 1):
    fake.fake_fail(b"{kind}", k)
    st = status(lambda: B200Backend(c, precision="{precision}").close())
    assert st == capi.SPO_ERR_OOM, (k, st)
    assert not live(), (k, live())
""")


def test_a_step_is_one_graph_and_says_so_when_it_is_not(run):
    """describe() names the graph; new arguments of the kernels are captured again, also after a profiled stretch; a
    capture that fails leaves launches one by one and its reason."""
    run("""
with B200Backend(case(), precision="mixed") as be:
    assert be.describe().endswith(" graph=1"), be.describe()
    n = fake.fake_launches(b"graph")
    be.propagate_analysis_step()
    assert fake.fake_launches(b"graph") == n + 1
    be.profile(True)
    be.test_wait_timeout(100, 16)
    be.test_wait_timeout(0, 0)
    be.propagate_analysis_step()
    be.profile(False)
    be.propagate_analysis_step()
    assert fake.fake_launches(b"graph") == n + 2, be.describe()
fake.fake_fail(b"capture", 1)
with B200Backend(case(), precision="mixed") as be:
    n, k = fake.fake_launches(b"graph"), fake.fake_launches(b"potential5")
    assert " graph=0 (" in be.describe(), be.describe()
    be.propagate_analysis_step()
    assert fake.fake_launches(b"graph") == n and fake.fake_launches(b"potential5") > k
assert not live()
""")


@pytest.mark.parametrize("env", [{}, {"FAKE_NO_MANAGED_ACCESS": "1"}])
def test_a_wait_that_gave_up_is_reported_by_every_call_that_runs_the_kernels(run, env):
    run("""
with B200Backend(case(), precision="mixed") as a, B200Backend(case(), precision="mixed") as b:
    fake.fake_raise(b"potential5", 1)
    assert status(lambda: a.apply_stage(capi.STAGE_POTENTIAL)) == capi.SPO_ERR_TIMEOUT
    with Ensemble([a, b]) as both:  # the stand-in runs a graph's kernels when it is captured
        fake.fake_raise(b"", 0)
        assert status(both.propagate_analysis_step) == capi.SPO_ERR_TIMEOUT
    assert status(a.propagate_analysis_step) == status(b.propagate_analysis_step) == capi.SPO_OK
assert not live(), live()
""", env)


@pytest.mark.parametrize("call", ["train", "gradients", "predict"])
def test_a_network_works_on_after_a_call_that_ran_out_of_memory(run, call):
    """Every allocation of a call's work space failing once: the status says so, and a smaller call then makes all of its
    own, as it does on a network that never failed (no buffer is taken for one that was not made)."""
    run(f"""
rng = np.random.default_rng(1)
x, y = rng.uniform(-1, 1, (1024, 12)).astype(np.float32), np.zeros(1024, np.float32)
calls = dict(train=lambda net, n: net.train(x[:n], y[:n], epochs=1, batch=n),
             gradients=lambda net, n: net.gradients(x[:n], y[:n]), predict=lambda net, n: net.predict(x[:n]))
go = calls["{call}"]
with Mlp(12, 128, 3) as net:
    go(net, 128)
    want = live()
with Mlp(12, 128, 3) as net:
    n = fake.fake_calls(b"malloc")
    go(net, 1024)
    n = fake.fake_calls(b"malloc") - n
assert n > 1 and not live()
for k in range(1, n + 1):
    with Mlp(12, 128, 3) as net:
        fake.fake_fail(b"malloc", k)
        assert status(lambda: go(net, 1024)) == capi.SPO_ERR_OOM, k
        go(net, 128)
        assert live() == want, (k, live(), want)
    assert not live(), k
""")


def test_what_a_network_keeps_for_the_next_call_is_bounded(run):
    """64 MiB for the points of predictions and 64 MiB for a training set, also after a call that failed."""
    run("""
n = 300001
x, y = np.ones((n, 64), np.float32), np.zeros(n, np.float32)
with Mlp(64, 64, 1) as net:
    net.predict(x[:128])
    before = fake.fake_bytes(b"malloc")
    k = fake.fake_launches(b"mlp_predict_kernel")
    net.predict(x)
    assert fake.fake_launches(b"mlp_predict_kernel") - k == 2
    assert 0 < fake.fake_bytes(b"malloc") - before <= 64 << 20, fake.fake_bytes(b"malloc") - before
with Mlp(64, 64, 1) as net:
    net.train(x[:128], y[:128], epochs=1, batch=128)
    before = fake.fake_bytes(b"malloc")
    net.train(x, y, epochs=1, batch=128)
    assert fake.fake_bytes(b"malloc") - before <= 64 << 20
    fake.fake_fail(b"malloc", 3)  # the third buffer of the training set
    assert status(lambda: net.train(x, y, epochs=1, batch=128)) == capi.SPO_ERR_OOM
    assert fake.fake_bytes(b"malloc") - before <= 64 << 20
""")


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("env", [{}, {"SPO_B200_BALANCED": "1"}, {"SPO_B200_PERSISTENT": "1"}, {"SPO_B200_KERNELS": "v1"},
                                 {"SPO_B200_PFA": "0"}])
@pytest.mark.parametrize("nz,nr,nx,ny", [(128, 48, 16, 16), (90, 36, 10, 10), (32, 27, 6, 4), (512, 24, 8, 8)])
def test_describe_names_the_kernels_that_run(run, nz, nr, nx, ny, env, precision):
    """The names of an analysis step's kinetic passes against the kernels that a step launches."""
    run(f"""
c = workload.config_case(dict(nz={nz}, nr={nr}, nx={nx}, ny={ny}, j_max=1, mj_max=1, nz_specular={nz}, nz_potential=2))
families = ("kin_kernel", "axis2_kernel", "axis2b_kernel", "axis2p_kernel", "axis2pfa_kernel", "xy2_kernel", "xy2p_kernel",
            "xy_pass_kernel")
with B200Backend(c, precision="{precision}") as be:
    be.profile(True)  # launch by launch
    before = [fake.fake_launches(f.encode()) for f in families]
    be.propagate_analysis_step()
    ran = {{f for f, b in zip(families, before) if fake.fake_launches(f.encode()) > b}}
    text = be.describe()
fields = dict(w.split("=", 1) for w in text.split() if "=" in w)
named = {{fields[k].split("<")[0].split("(")[0] + "_kernel" for k in ("z", "r", "xy")}}
assert named - {{"axis_pass_kernel"}} == ran, (named, ran, text)
assert (fields["balanced"] == "1") == ("axis2b_kernel" in ran) and (fields["persistent"] != "") == bool(ran & {{"axis2p_kernel", "xy2p_kernel"}}), text
""", env)


def test_odd_numbers_of_lanes_take_the_kernels_that_load_them_one_by_one(run):
    """n_rot 81 (J 8) and 169 (J 12) against 100 (J 9): the pairs of kin_kernel need even rows; the smallest cells only where
    long rows do not fit L2; and more points than the other kernels have block rows stay where they run."""
    run("""
def names(precision, n, j, nz=24, nr=24):
    c = workload.config_case(dict(nz=nz, nr=nr, nx=n, ny=n, j_max=j, mj_max=j, nz_specular=nz, nz_potential=1))
    with B200Backend(c, precision=precision) as be:
        return {k: v.split("<")[0] for k, v in (w.split("=", 1) for w in be.describe().split() if "=" in w) if k in "z r xy"}
for n in (8, 12, 16):
    assert names("mixed", n, 9)["xy"] == "kin" and names("mixed", n, 8)["xy"] in ("xy2", "xy2p"), n
assert names("mixed", 6, 8)["xy"] == "kin" and names("mixed", 10, 8)["xy"] == "kin"
for precision, nz in (("fp64", 160), ("mixed", 320)):  # 150 MB of 4 x 4 cells
    assert names(precision, 4, 8, nz, 24)["xy"] == "kin" and names(precision, 4, 12, 24, 24)["xy"] == "kin", precision
    assert names(precision, 4, 12, nz, 24)["xy"] == "xy2", precision
assert names("fp64", 8, 12)["xy"] == "kin"
assert names("mixed", 8, 2)["xy"] == "kin" and names("mixed", 16, 0)["xy"] == "kin" and names("mixed", 16, 2)["xy"] == "xy2p"
assert names("mixed", 12, 2, 2048, 33)["xy"] == "kin"  # 67584 points
assert names("mixed", 5, 8, 128, 48) == {"z": "kin", "r": "axis2pfa", "xy": "kin"}  # 48 r points: even rows for Z
assert names("mixed", 5, 8, 128, 27)["z"] == "axis2b" and names("mixed", 5, 9, 128, 27)["z"] == "kin"
assert names("fp64", 5, 8, 128, 48) == {"z": "kin", "r": "kin", "xy": "kin"}
""")


COPIES = """
def packet(be, c, seed):
    psi = np.random.default_rng(seed).standard_normal(c.psi_shape).astype(np.float32) + 0j
    be.read_wave_packet(psi, None)
    return np.array_equal(be.wave_packet_on_host()[0], psi)
big, mid, small = (case(nz=nz, nr=32, nx=8, ny=8, j=5, nzp=1) for nz in (64, 16, 4))
mib = [c.nz * c.nr * c.nx * c.ny * c.n_rot * 16 / 2**20 for c in (big, mid, small)]
assert mib == [72.0, 18.0, 4.5], mib
"""


def test_copies_go_on_without_pinned_memory(run):
    """A packet of 72 MiB where the pinned buffers or their streams cannot be had: by plain copies, nothing left behind."""
    run(COPIES + """
for kind, nth in ((b"host", 1), (b"stream", 2), (b"event", 3)):
    with B200Backend(big, precision="fp64") as be:
        fake.fake_fail(kind, nth)
        assert packet(be, big, 1), kind
        assert fake.fake_live(b"host") == 1, kind  # asked for again by the second copy
    assert not live(), live()
x, calls = np.ones((1500000, 12), np.float32), fake.fake_calls(b"host")
with Mlp(12, 64, 1) as net:
    fake.fake_fail(b"host", 1)
    net.predict(x)
    assert fake.fake_calls(b"host") == calls + 1 and fake.fake_live(b"host") == 0
""")


def test_pinned_buffers_are_made_when_the_copies_pay_for_them(run):
    """Not for one packet of 18 MiB up and down, but at the fourth such copy; at once for a large one; not for small ones
    however often; and shared by the handles of the device."""
    run(COPIES + """
with B200Backend(mid, precision="fp64") as be:
    assert packet(be, mid, 1) and fake.fake_calls(b"host") == 0
    assert packet(be, mid, 2) and fake.fake_calls(b"host") == 1
    with B200Backend(mid, precision="fp64") as other, B200Backend(big, precision="fp64") as third:
        assert packet(other, mid, 3) and packet(third, big, 4) and fake.fake_calls(b"host") == 1
with B200Backend(big, precision="fp64") as be:
    assert packet(be, big, 5) and fake.fake_calls(b"host") == 2
with B200Backend(small, precision="fp64") as be:
    assert all(packet(be, small, k) for k in range(40)) and fake.fake_calls(b"host") == 2
assert not live()
""")


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_a_handle_holds_no_tables_of_kernels_it_does_not_launch(run, precision):
    """The same potential kernel by default and named: only the named one can fall back to others, whose tables it holds."""
    run(f"""
c = case(j=15, nx=8, ny=8)
out = []
for kernels in (None, "v5"):
    if kernels:
        os.environ["SPO_B200_KERNELS"] = kernels
    with B200Backend(c, precision="{precision}") as be:
        out.append((be.device_bytes(), [w for w in be.describe().split() if w.startswith("potential=")], fake.fake_live(b"malloc")))
(few, a, n), (all_tables, b, m) = out
assert a == b and few < all_tables and n < m, out
""")
