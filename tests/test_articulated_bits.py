"""The articulated step against recorded results, bit for bit.

A contact world amplifies one ulp into another contact decision (a point kept
or dropped) now and then, so a change of rounding -- an expression contracted
in another order, a division turned into a product -- shows as a few
environments far off and not as an error that a tolerance could bound.  The
records (tests/golden/make_articulated_bits.py) hold the arithmetic."""

from __future__ import annotations

from pathlib import Path

import numpy as np
import pytest

import numi_lab_b200 as nb

pytestmark = pytest.mark.gpu

GOLDEN = Path(__file__).resolve().parent / "golden" / "articulated_bits.npz"
SEED = 11
# Source, precision, solver, control steps.
CASES = {
    "tree29_fp32": ("tree29", "fp32", None, 6),
    "tree29_fp64_inertia": ("tree29", "fp64-inertia", None, 3),
    "tree29_compensated": ("tree29", "compensated", None, 3),
    "tree29_quality": ("tree29", "fp32", "quality_newton", 1),
    "chain7_fp32": ("chain7", "fp32", None, 20),
    "chain7_fp64_inertia": ("chain7", "fp64-inertia", None, 20),
}


def rollout(name, q, v, actions):
    import torch

    source, precision, solver, _ = CASES[name]
    options = {"substeps": 1, "control_dt": 0.005} if source == "chain7" else {"substeps": 4, "velocity_iterations": 8, "control_dt": 0.02}
    with nb.World(source, len(q), seed=SEED, precision=precision, **options) as w:
        if solver:
            w.set_solver(solver)
        w.reset(SEED)
        w.set_state(q, v)
        _, status, _ = w.step(torch.from_numpy(actions).cuda(), wait=True)
        assert int(status.abs().sum()) == 0
        return w.state()[:2]


@pytest.mark.parametrize("name", sorted(CASES))
def test_end_states_are_the_recorded_bits(cuda_device, name):
    golden = np.load(GOLDEN)
    q1, v1 = rollout(name, *(golden[f"{name}_{k}"] for k in ("q", "v", "actions")))
    np.testing.assert_array_equal(q1, golden[f"{name}_q1"])
    np.testing.assert_array_equal(v1, golden[f"{name}_v1"])
