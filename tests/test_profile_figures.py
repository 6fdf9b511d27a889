"""bench.py reports counters of a committed summary only while they were
counted on the kernel whose time it reports them with."""

from __future__ import annotations

import shutil

import bench


def _summary(tmp_path, fingerprint):
    path = tmp_path / "summary.md"
    path.write_text(f"| traffic | 1 |\n\nkernel_sources: {fingerprint}\nwarp_instructions_per_env_step: 123\nbroken: figure\n")
    return path


def test_figures_of_the_present_kernel_are_read(tmp_path):
    path = _summary(tmp_path, bench._kernel_fingerprint())
    assert bench._profile_value("warp_instructions_per_env_step", path) == 123.0
    assert bench._profile_value("broken", path) is None and bench._profile_value("absent", path) is None


def test_figures_of_another_kernel_are_not(tmp_path):
    assert bench._profile_value("warp_instructions_per_env_step", _summary(tmp_path, "0123456789abcdef")) is None
    unmarked = tmp_path / "unmarked.md"
    unmarked.write_text("warp_instructions_per_env_step: 123\n")
    assert bench._profile_value("warp_instructions_per_env_step", unmarked) is None


def test_the_fingerprint_follows_code_and_not_comments(tmp_path):
    for name in bench.KERNEL_SOURCES:
        shutil.copy(bench.ROOT / "numi_lab_b200" / "csrc" / name, tmp_path / name)
    changed = tmp_path / bench.KERNEL_SOURCES[1]
    changed.write_text("// a remark\n" + changed.read_text())
    assert bench._kernel_fingerprint(tmp_path) == bench._kernel_fingerprint()
    changed.write_text(changed.read_text() + "int more;\n")
    assert bench._kernel_fingerprint(tmp_path) != bench._kernel_fingerprint()
