"""Generates tests/golden/articulated_bits.npz: start states, actions and the
exact FP32 end states of short rollouts on one B200, per world and mode
(tests/test_articulated_bits.py).  The committed file was recorded with the
single-sweep forward kinematics and the divisions by L_kk in the velocity
sweep; it is recorded again only when the arithmetic of the articulated step
changes on purpose.

Run from the repository root on a GPU:  python tests/golden/make_articulated_bits.py
"""

from __future__ import annotations

import sys
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parents[2]
sys.path.insert(0, str(ROOT))
sys.path.insert(0, str(ROOT / "tests"))

import numi_lab_b200 as nb  # noqa: E402

from test_articulated_bits import CASES, GOLDEN, rollout  # noqa: E402

SEED, ENVS = 11, 48


def main() -> None:
    rng = np.random.default_rng(2026)
    data = {}
    for name, (source, _, _, steps) in CASES.items():
        q, v, _ = nb.sample_reset(source, SEED, 5, 0, ENVS)
        q, v = np.ascontiguousarray(q, np.float32), (v + rng.normal(0.0, 0.1, v.shape)).astype(np.float32)
        if source == "tree29":  # half of them pressed onto the ground, so that feet and proxies touch
            q[::2, 2] -= 0.02
        width = nb.compile_model(source, SEED).world.action_count
        actions = rng.normal(0.0, 0.3, (steps, ENVS, width)).astype(np.float32)
        q1, v1 = rollout(name, q, v, actions)
        data.update({f"{name}_q": q, f"{name}_v": v, f"{name}_actions": actions, f"{name}_q1": q1, f"{name}_v1": v1})
    np.savez_compressed(GOLDEN, **data)


if __name__ == "__main__":
    main()
