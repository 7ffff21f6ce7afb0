"""Barriers of the FP32 hop loops: the kernels' own source compiled for the
host, a host thread per device thread (host_threads/device.h), under
ThreadSanitizer, which reports any two accesses of shared memory that no
barrier orders."""
import os
import re
import shutil
import subprocess

import pytest

from conftest import REPO

HERE = os.path.join(REPO, "tests", "host_threads")
CSRC = os.path.join(REPO, "kmc_dn_gb300", "csrc")
HOST = {"ex2.approx": "y = exp2f(x);", "rcp.approx": "y = 1.0f / x;", "rsqrt.approx": "y = 1.0f / sqrtf(x);",
        "globaltimer": "t = 0;"}
LAUNCHES = ["slices of 4, one temperature", "slices of 8, positions, recorded", "block of 64, recorded",
            "block of 64, positions, no stored sums", "block of 256, positions",
            "slices of 16, sites four a step, recorded", "whole warp, sites two a step"]


def _cuda_include():
    nvcc = os.path.realpath(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc")
    return os.path.join(os.path.dirname(os.path.dirname(nvcc)), "include")


def _host_source(text):
    """Device source as the host compiler takes it: launches as calls, PTX as
    its value, shared memory as storage that the threads share."""
    text = re.sub(r"<<<.*?>>>", "", text, flags=re.S)
    for op, value in HOST.items():
        text = re.sub(r'asm( volatile)?\("[^"]*%s[^;]*;[^;]*;' % re.escape(op), value, text)
    text = re.sub(r"extern __shared__ __align__\(16\) (\w+) (\w+)\[\];",
                  r"\1 *\2 = reinterpret_cast<\1 *>(dynamic_smem);", text)
    text = re.sub(r"\b__shared__\b", "static", text)
    return text.replace('"../../include/kmc_dn_gb300.h"', '"%s/include/kmc_dn_gb300.h"' % REPO)


def _compile(folder, source, out, *flags, sanitize="thread"):
    cmd = ["g++", "-std=c++20", "-O1", "-g", f"-fsanitize={sanitize}", "-pthread", "-w", *flags, source, "-o", out]
    return subprocess.run(cmd, capture_output=True, text=True, cwd=folder)


def _sources(folder):
    for name in os.listdir(CSRC):
        if name.endswith((".cuh", ".h")):
            with open(os.path.join(CSRC, name)) as f:
                (folder / name).write_text(_host_source(f.read()))
    return ["-I", str(folder), "-I", HERE, "-I", _cuda_include()]


@pytest.fixture(scope="module")
def engine(tmp_path_factory):
    folder = tmp_path_factory.mktemp("host_threads")
    probe = folder / "probe.cpp"
    probe.write_text("#include <thread>\nint x;\nint main() { std::thread a([] { x = 1; }), b([] { x = 2; }); "
                     "a.join(); b.join(); }\n")
    if not shutil.which("g++") or _compile(folder, str(probe), "probe").returncode or \
            "data race" not in subprocess.run([str(folder / "probe")], capture_output=True, text=True).stderr:
        pytest.skip("no g++ with a working ThreadSanitizer")
    r = _compile(folder, os.path.join(HERE, "engine.cpp"), "engine", *_sources(folder))
    assert r.returncode == 0, r.stderr[-4000:]
    return str(folder / "engine")


@pytest.mark.parametrize("launch", range(len(LAUNCHES)), ids=LAUNCHES)
def test_shared_memory_is_ordered(engine, launch):
    r = subprocess.run([engine, str(launch)], capture_output=True, text=True, timeout=600)
    races = re.findall(r"SUMMARY: ThreadSanitizer: (.*)", r.stderr)
    assert not races, "\n".join(sorted(set(races)))
    assert r.returncode == 0, r.stderr[-2000:]


def test_debug_build_checks_the_runs(tmp_path):
    """-DKMC_DEBUG_CHECKS: a run that leaves the state's pairs is refused before
    its records are read, and the launches above pass their checks (with the
    address sanitizer on their shared memory)."""
    if not shutil.which("g++"):
        pytest.skip("no g++")
    r = _compile(tmp_path, os.path.join(HERE, "engine.cpp"), "checked", "-DKMC_DEBUG_CHECKS", *_sources(tmp_path),
                 sanitize="address")
    assert r.returncode == 0, r.stderr[-4000:]
    for launch in range(len(LAUNCHES) + 1):
        r = subprocess.run([str(tmp_path / "checked"), str(launch)], capture_output=True, text=True, timeout=600)
        assert r.returncode == 0 and "error" not in r.stderr, (launch, r.stderr[-2000:])
