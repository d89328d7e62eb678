"""Failure detection of the bounded device-side waits, without a GPU fault (needs a B200).

potential5 and potential6 move each item's data by bulk asynchronous copies whose completion is counted in
bytes on an mbarrier, and every wait on a barrier is bounded. spo_test_wait_timeout makes every item's
first barrier announce 16 bytes more than its copies deliver: every copy is valid and lands, but the
barrier's phase cannot complete. Each block's wait then gives up after a short poll limit, the block sets
the device error flag, waits (bounded) for its own work in flight, frees its tensor memory and leaves, and
the step returns SPO_ERR_TIMEOUT with the context intact. After the hook is cleared and the wave packet is
uploaded again, the next step is bitwise the step of a handle that never failed.
"""

import numpy as np
import pytest

from test_gpu_kernels import make

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernels", ["v5", "v6"])
def test_a_wait_that_gives_up_returns_timeout_and_the_handle_recovers(kernels):
    from spo_b200 import capi, workload
    case = workload.config_case({"nz": 24, "nr": 16, "nx": 8, "ny": 8, "j_max": 15, "mj_max": 15,
                                 "nz_specular": 64, "nz_potential": 14})
    rng = np.random.default_rng(31)
    psi0 = rng.standard_normal(case.psi_shape) + 1j * rng.standard_normal(case.psi_shape)
    chi0 = rng.standard_normal(case.chi_shape) + 1j * rng.standard_normal(case.chi_shape)
    with make(case, kernels, "mixed") as ref:
        assert f"potential=potential{kernels[1]}" in ref.describe(), ref.describe()
        ref.read_wave_packet(psi0, chi0)
        ref.propagate_analysis_step()
        expected = ref.wave_packet_on_host()
    with make(case, kernels, "mixed") as be:
        be.read_wave_packet(psi0, chi0)
        be.test_wait_timeout(1 << 16, 16)
        with pytest.raises(capi.B200Error) as err:
            be.propagate_analysis_step()
        assert err.value.status == capi.SPO_ERR_TIMEOUT, str(err.value)
        assert "gave up" in str(err.value)
        be.test_wait_timeout(0, 0)
        be.read_wave_packet(psi0, chi0)
        be.propagate_analysis_step()
        psi, chi = be.wave_packet_on_host()
    assert np.array_equal(psi, expected[0]) and np.array_equal(chi, expected[1])


def test_unmatched_bytes_must_be_a_multiple_of_16():
    from spo_b200 import capi, workload
    case = workload.config_case({"nz": 16, "nr": 16, "nx": 4, "ny": 4, "j_max": 3, "mj_max": 3,
                                 "nz_specular": 32, "nz_potential": 8})
    with make(case, "v5", "mixed") as be:
        with pytest.raises(capi.B200Error) as err:
            be.test_wait_timeout(100, 8)
        assert err.value.status == capi.SPO_ERR_INVALID


@pytest.mark.parametrize("failing", [(0,), (1,), (0, 2)])
def test_an_ensemble_reports_a_wait_that_gave_up_and_its_members_recover(failing):
    """The graph holds the arguments its members had when it was made."""
    from spo_b200 import Ensemble, capi, workload
    case = workload.config_case({"nz": 24, "nr": 16, "nx": 4, "ny": 4, "j_max": 7, "mj_max": 7,
                                 "nz_specular": 64, "nz_potential": 14})
    rng = np.random.default_rng(5)
    psi0 = rng.standard_normal(case.psi_shape) + 1j * rng.standard_normal(case.psi_shape)
    chi0 = rng.standard_normal(case.chi_shape) + 1j * rng.standard_normal(case.chi_shape)
    members = [make(case, None, p) for p in ("mixed", "mixed", "mixed", "fp64")]
    try:
        members[0].read_wave_packet(psi0, chi0)
        members[0].propagate_analysis_step()
        expected = members[0].wave_packet_on_host()
        for k in failing:
            members[k].test_wait_timeout(1 << 16, 16)
        with Ensemble(members) as ensemble:
            for _ in range(2):  # the flags are cleared by the report, and set again by the next step
                with pytest.raises(capi.B200Error) as err:
                    ensemble.propagate_analysis_step()
                assert err.value.status == capi.SPO_ERR_TIMEOUT and f"member {failing[0]}:" in str(err.value), str(err.value)
        for k in failing:
            members[k].test_wait_timeout(0, 0)
        with Ensemble(members) as ensemble:
            for m in members:
                m.read_wave_packet(psi0, chi0)
            ensemble.propagate_analysis_step()
            for m in members[:3]:
                psi, chi = m.wave_packet_on_host()
                assert np.array_equal(psi, expected[0]) and np.array_equal(chi, expected[1])
    finally:
        for m in members:
            m.close()


def test_a_single_operator_reports_a_wait_that_gave_up():
    from spo_b200 import capi, workload
    case = workload.config_case({"nz": 24, "nr": 16, "nx": 4, "ny": 4, "j_max": 7, "mj_max": 7,
                                 "nz_specular": 64, "nz_potential": 14})
    with make(case, None, "mixed") as be:
        be.test_wait_timeout(1 << 16, 16)
        with pytest.raises(capi.B200Error) as err:
            be.apply_stage(capi.STAGE_POTENTIAL)
        assert err.value.status == capi.SPO_ERR_TIMEOUT
        be.test_wait_timeout(0, 0)
        be.apply_stage(capi.STAGE_POTENTIAL)
        be.propagate_analysis_step()


def test_a_training_step_that_failed_changes_nothing_and_the_network_recovers():
    """With a poll limit of 0 every wait for the tensor cores gives up at once (the products in flight are then waited for
    before a block leaves). The parameters and Adam's state stay as they were, so the training that follows is bitwise
    that of a network that never failed."""
    from spo_b200 import capi
    from spo_b200.mlp import Mlp
    rng = np.random.default_rng(3)
    x = rng.uniform(-1.0, 1.0, (2048, 12)).astype(np.float32)
    y = np.sin(x.sum(axis=1)).astype(np.float32)
    results = []
    for failing in (False, True):
        with Mlp(12, 128, 3, seed=4) as net:
            net.train(x, y, epochs=1, batch=512, seed=1)
            if failing:
                before = net.get_parameters()
                net.test_wait_timeout(0)
                for call in (lambda: net.train(x, y, epochs=1, batch=512, seed=2), lambda: net.gradients(x, y),
                             lambda: net.predict(x)):
                    with pytest.raises(capi.B200Error) as err:
                        call()
                    assert err.value.status == capi.SPO_ERR_TIMEOUT, str(err.value)
                net.test_wait_timeout(-1)
                assert np.array_equal(net.get_parameters(), before)
            loss = net.train(x, y, epochs=1, batch=512, seed=5)
            results.append((loss, net.get_parameters(), net.predict(x)))
    assert results[0][0] == results[1][0]
    assert all(np.array_equal(a, b) for a, b in zip(results[0][1:], results[1][1:]))


def test_a_prediction_that_gives_up_anywhere_leaves_the_next_one_intact():
    """Poll limits from 0 upwards end a block's work at different waits: before its weights, between two products, before a
    layer's end. Each call either succeeds or says that it timed out, and a block that leaves has nothing in flight that
    could reach the shared memory of the next."""
    from spo_b200 import capi
    from spo_b200.mlp import Mlp
    x = np.random.default_rng(6).uniform(-1.0, 1.0, (100000, 12)).astype(np.float32)
    with Mlp(12, 256, 4, seed=4) as net:
        want = net.predict(x)
        outcomes = set()
        for polls in [0, 1, 2, 3, 4, 6, 8, 12, 16, 24, 32, 64, 128, 256] * 3:
            net.test_wait_timeout(polls)
            try:
                assert np.array_equal(net.predict(x), want)
                outcomes.add("done")
            except capi.B200Error as e:
                assert e.status == capi.SPO_ERR_TIMEOUT, str(e)
                outcomes.add("timeout")
            net.test_wait_timeout(-1)
            assert np.array_equal(net.predict(x), want), polls
        assert "timeout" in outcomes, outcomes
