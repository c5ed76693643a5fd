"""Small programs linked to the library, for what it decides on the host from a call's shape alone."""

from __future__ import annotations

import json
import pathlib
import shutil
import subprocess

import pytest

from deformops_b200._build import LIB_PATH, NVCC_FLAGS, CSRC, build_library


def host_program(source: str, where: pathlib.Path):
    """``run(call, ...)`` of the program: it gets the calls' whole numbers, and prints a JSON line for each."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not pathlib.Path(nvcc).exists():
        pytest.skip("nvcc not installed")
    build_library()
    path, program = where / "program.cu", where / "program"
    path.write_text(source)
    done = subprocess.run([nvcc, *NVCC_FLAGS, f"-I{CSRC}", str(path), "-o", str(program), str(LIB_PATH),
                           "-Xlinker", f"-rpath={LIB_PATH.parent}"], capture_output=True, text=True)
    assert done.returncode == 0, done.stderr

    def run(*calls):
        done = subprocess.run([str(program), *[str(int(x)) for call in calls for x in call]],
                              capture_output=True, text=True)
        assert done.returncode == 0, done.stderr
        return [json.loads(line) for line in done.stdout.splitlines()]

    return run
