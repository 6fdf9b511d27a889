"""Launch shapes follow the environment count (and, for free bodies, the body
count: warps per environment, shared memory); no arithmetic does.  The
first environments of a large world therefore end on the same bits as the
same environments in a small one, on both sides of every rule, and also when
a substep's contacts do not fit the small shape's shared memory."""

from __future__ import annotations

import numpy as np
import pytest

import numi_lab_b200 as nb

pytestmark = pytest.mark.gpu

FEW = 6  # four warps per environment


def _run(source, seed, envs, q, v, steps):
    import torch

    with nb.World(source, envs, substeps=4, velocity_iterations=8, control_dt=0.02, seed=seed) as w:
        reps = -(-envs // FEW)
        w.set_state(np.tile(q, (reps, 1))[:envs], np.tile(v, (reps, 1))[:envs])
        _, status, _ = w.step(torch.zeros((steps, envs, 0), device="cuda"), wait=True)
        assert int(status.abs().sum()) == 0
        q1, v1, table = w.state()
        return q1[:FEW], v1[:FEW], table[:FEW]


def _same(a, b):
    for name, x, y in zip(("q", "v", "manifolds"), a, b):
        np.testing.assert_array_equal(x, y, err_msg=name)


# One, two and four warps: small and large worlds below and above 592 and 1184
# environments (four and eight per SM).
@pytest.mark.parametrize("source,bodies,envs", [("pile", 9, 600), ("pile", 9, 1190), ("pile", 28, 1190), ("pile", 29, 600),
                                                ("pile", 64, 1190), ("cylinder_pile", 23, 600), ("cylinder_pile", 23, 1190),
                                                ("hull_pile", 29, 600)])
def test_every_launch_shape_gives_the_same_bits(cuda_device, source, bodies, envs):
    seed = nb.world.pile_seeds_by_body_count([bodies])[bodies]
    q, v, _ = nb.sample_reset(source, seed, 7, 0, FEW)
    few = _run(source, seed, FEW, q, v, 12)
    many = _run(source, seed, envs, q, v, 12)
    _same(few, many)


def test_contacts_beyond_the_shared_arrays(cuda_device):
    """28 upright bodies drawn together until they make about 160 contacts:
    more than the 125 that the one-warp shape of a support-mapped world this
    size keeps in shared memory (its 2800 words less the 1670 of the rest,
    nine words per contact)."""

    bodies, envs, shrink = 28, 1190, 0.25
    seed = nb.world.pile_seeds_by_body_count([bodies])[bodies]
    q, v, _ = nb.sample_reset("pile_gjk", seed, 7, 0, FEW)  # three layers
    q = q.reshape(FEW, bodies, 7).copy()
    q[:, :, :2] *= shrink
    q[:, :, 2] = 0.05 + (q[:, :, 2] - q[:, :, 2].min()) * shrink
    q[:, :, 3:] = (0.0, 0.0, 0.0, 1.0)
    results = []
    for n in (FEW, envs):
        with nb.World("cylinder_pile", n, substeps=1, velocity_iterations=8, control_dt=0.005, seed=seed) as w:
            reps = -(-n // FEW)
            w.set_state(np.tile(q.reshape(FEW, -1), (reps, 1))[:n], np.tile(np.zeros_like(v), (reps, 1))[:n])
            out = w.advance_host(np.zeros((1, n, 0), np.float32))
            assert (out["status"] == 0).all() and out["contacts"].min() > 125
            results.append(tuple(x[:FEW] for x in w.state()))
    _same(*results)


# Environments per CTA of the articulated kernel against one (a few
# environments): one CTA per SM past eight environments on each (1184), full
# CTAs of one resident wave and of two chains, the quality instance's three,
# and four, by the override, where the plan itself holds one.
@pytest.mark.parametrize("source,envs,precision,solver,per_cta,fixed", [
    ("tree29", 1190, "fp32", None, 9, False), ("tree29", 2368, "fp32", None, 16, False), ("tree29", 2400, "fp32", None, 16, False),
    ("tree29", 1190, "fp32", "quality_newton", 3, False), ("tree29", 1190, "fp64-inertia", None, 4, True),
    ("tree29", 1190, "compensated", None, 4, True), ("chain7", 1190, "fp32", None, 4, True)])
def test_articulated_launches_give_the_same_bits(cuda_device, monkeypatch, source, envs, precision, solver, per_cta, fixed):
    import torch

    options = {"substeps": 1, "control_dt": 0.005} if source == "chain7" else {"substeps": 4, "velocity_iterations": 8, "control_dt": 0.02}
    steps = 2 if solver else 10
    ends = []
    for n in (FEW, envs):
        if fixed and n == envs:
            monkeypatch.setenv("NUMI_B200_STEP_WARPS_PER_BLOCK", str(per_cta))
        with nb.World(source, n, seed=5, precision=precision, **options) as w:
            if solver:
                w.set_solver(solver)
            assert w.launch_shape()[0] == (1 if n == FEW else per_cta)
            gen = np.random.default_rng(3)
            acts = gen.normal(0.0, 0.3, (steps, FEW, w.action_count)).astype(np.float32)
            acts = np.tile(acts, (1, -(-n // FEW), 1))[:, :n]
            q, v, _ = nb.sample_reset(source, 5, 5, 0, FEW)
            w.set_state(np.tile(q, (-(-n // FEW), 1))[:n], np.tile(v, (-(-n // FEW), 1))[:n])
            _, status, _ = w.step(torch.from_numpy(np.ascontiguousarray(acts)).cuda(), wait=True)
            assert int(status.abs().sum()) == 0
            q1, v1, m = w.state()
            ends.append((q1[:FEW], v1[:FEW], np.frombuffer(bytes(m), np.uint8)[:FEW * w.pair_count * 224]))
    _same(*ends)


def _sms():
    import torch

    return torch.cuda.get_device_properties(0).multi_processor_count


def _shape(envs, **options):
    with nb.World("tree29", envs, substeps=4, velocity_iterations=8, control_dt=0.02, **options) as w:
        return w.launch_shape()


def test_the_reported_shape_is_the_launched_one(cuda_device):
    """One environment per CTA up to eight per SM, then one CTA per SM up to
    a resident wave, then two chains of full CTAs."""

    sms = _sms()
    full = 16  # environments per CTA and per SM at full residency
    assert _shape(1)[0] == _shape(FEW)[0] == _shape(8 * sms)[0] == 1
    assert _shape(8 * sms + 1) == (9, 9)
    assert _shape(full * sms) == (full, full)
    assert _shape(full * sms + 1) == (full, full)
    assert _shape(FEW)[1] >= 8  # a spread launch is resident at once


def test_a_fixed_cta_size_is_read_at_creation(cuda_device, monkeypatch):
    options = {"substeps": 4, "velocity_iterations": 8, "control_dt": 0.02}
    name = "NUMI_B200_STEP_WARPS_PER_BLOCK"
    monkeypatch.delenv(name, raising=False)
    with nb.World("tree29", FEW, **options) as spread:
        monkeypatch.setenv(name, "4")
        with nb.World("tree29", FEW, **options) as fixed:
            assert (spread.launch_shape()[0], fixed.launch_shape()[0]) == (1, 4)
            monkeypatch.delenv(name)
            assert (spread.launch_shape()[0], fixed.launch_shape()[0]) == (1, 4)
