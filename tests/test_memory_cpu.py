"""Memory, copies and timers of the library against a CUDA runtime made of host code (tests/cpp/fake_cuda_runtime.h): what two
GPUs, failing calls and exceptions do to them can be had without either."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "superkmeans_b200", "csrc")
CPP = os.path.join(ROOT, "tests", "cpp")
SOURCES = {"memory_check": ["memory.cu"], "copies_check": ["memory.cu", "host_copy.cu"], "timers_check": ["memory.cu", "phase_timers.cu"]}


def _cuda_include():
    nvcc = os.environ.get("NVCC") or shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    return os.path.join(os.path.dirname(os.path.dirname(nvcc)), "include")


@pytest.fixture(scope="session")
def program(tmp_path_factory):
    made = {}

    def make(name):
        if name not in made:
            exe = str(tmp_path_factory.mktemp("fake_cuda") / name)
            cmd = ["/usr/bin/g++", "-std=c++17", "-O1", "-Wall", "-Wno-unknown-pragmas", "-fopenmp", "-I", _cuda_include(), "-x", "c++", os.path.join(CPP, name + ".cpp"),
                   os.path.join(CPP, "fake_cuda_runtime.cpp")] + [os.path.join(CSRC, s) for s in SOURCES[name]] + ["-o", exe, "-lpthread"]
            res = subprocess.run(cmd, capture_output=True, text=True)
            assert res.returncode == 0, res.stderr
            made[name] = exe
        return made[name]

    return make


@pytest.mark.parametrize("name,case", [("memory_check", "events_between_devices"), ("memory_check", "record_that_fails"), ("memory_check", "modes"), ("memory_check", "device_memory_that_is_short"), ("memory_check", "pinned_memory_that_is_short"),
                                       ("copies_check", "exception_behind_a_copy"), ("copies_check", "exception_behind_a_pinned_copy"), ("copies_check", "rows_arrive"), ("copies_check", "pieces_of_any_length"), ("copies_check", "device_memory"),
                                       ("timers_check", "many_calls"), ("timers_check", "nothing_unfinished_is_read")])
def test_with_a_runtime_of_host_code(program, name, case):
    res = subprocess.run([program(name), case], capture_output=True, text=True, timeout=120)
    assert res.returncode == 0 and "OK" in res.stdout, res.stdout + res.stderr


def test_workspace_cache_answers_what_was_set():
    from superkmeans_b200 import engine

    before = engine.workspace_cache()
    try:
        for mode in (1, 0, 2):
            engine.set_workspace_cache(mode)
            assert engine.workspace_cache() == mode
    finally:
        engine.set_workspace_cache(before)
    assert before == 2
