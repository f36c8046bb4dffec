"""Kernels' own sources on the CPU, every thread a fiber (tests/emulation/kernel_emulator.hpp): interleavings
that an idle GPU hardly ever shows."""

from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

EMULATION = Path(__file__).resolve().parent / "emulation"
FLAGS = ["-std=c++17", "-O2", "-ffp-contract=off", "-fno-strict-aliasing", "-Wall", "-Wextra", "-Wno-unknown-pragmas"]


def _build(source: Path, exe: Path, *flags: str) -> Path:
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    subprocess.run([cxx, *FLAGS, *flags, str(source), "-o", str(exe)], check=True)
    return exe


def _run(exe: Path, *args: str) -> None:
    out = subprocess.run([str(exe), *args], capture_output=True, text=True, timeout=600)
    assert out.returncode == 0, out.stderr[-2000:]


@pytest.fixture(scope="module")
def small_walks(tmp_path_factory):
    return _build(EMULATION / "small_walks.cpp", tmp_path_factory.mktemp("emulation") / "small_walks", "-DTMC_FAST_MASK=0")


def test_no_photon_is_lost_when_blocks_start_late(small_walks):
    """1 to 32 lanes a warp, blocks of 1 to 4 warps, some of them starting when others have long claimed
    their second photons."""
    _run(small_walks, "late_blocks")


def test_packets_walked_alone_through_thin_layers(small_walks):
    """Boundary after boundary, with nothing scored in between: the layer's tables are rewritten only when
    every lane of the warp has read the last one's."""
    _run(small_walks, "layer_changes")


def test_scores_that_are_no_numbers(small_walks):
    """A packet walked alone sums its scores as a lane does, also where each is no number (2^63)."""
    _run(small_walks, "no_numbers")


@pytest.mark.parametrize("case", ["lanes_apart", "sweep_lanes_apart"])
def test_lanes_of_a_warp_leave_the_step_loop_together(small_walks, case):
    """Lanes scheduled independently: each reads the block's counts of live lanes at its own time, while other
    warps write them."""
    _run(small_walks, case)


def test_gemm_roles_give_up_together(tmp_path):
    """Waits of the tensor-core GEMM that run out while some lanes of the warp see their barrier complete."""
    shutil.copy(EMULATION.parents[1] / "tissuemc_b200/csrc/gemm_tc.cuh", tmp_path / "gemm_tc.cuh")
    shutil.copy(EMULATION / "umma_stub.hpp", tmp_path / "umma.cuh")
    for header in ("cuda.h", "cuda_bf16.h"):
        (tmp_path / header).write_text("")
    _run(_build(EMULATION / "gemm_waits.cpp", tmp_path / "gemm_waits", f"-I{tmp_path}"))
