"""The order of the kernels' accesses to their shared variables, on the CPU:
the device code's own synchronisation (read from its sources, with the PTX
wrappers replaced by host stand-ins) runs on host threads."""
import re
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "cup2d_b200" / "csrc"
CPP = ROOT / "tests" / "cpp"


def host_source(name):
    """A device header without its includes and without the functions that
    wrap PTX (tests/cpp/cuda_threads.hpp has their stand-ins)."""
    text = re.sub(r"^#(include|pragma).*\n", "", (CSRC / name).read_text(), flags=re.M)
    functions = re.compile(r"^(?:template <[^>]*>\n)?__device__[^;{}]*\{\n.*?^\}\n", re.M | re.S)
    return functions.sub(lambda m: "" if re.search(r"\basm\b", m.group(0)) else m.group(0), text)


def build(tmp_path, source, includes, *flags):
    for inc, names in includes.items():
        (tmp_path / inc).write_text("".join(host_source(n) for n in names))
    exe = tmp_path / source.removesuffix(".cpp")
    subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-pthread", *flags, "-I", str(tmp_path), "-I", str(CPP),
                    str(CPP / source), "-o", str(exe)], check=True)
    return exe


def sanitizer_runs(tmp_path):
    src, exe = tmp_path / "probe.cpp", tmp_path / "probe"
    src.write_text("#include <thread>\nint x; int main() { std::thread a([] { ++x; }), b([] { ++x; }); "
                   "a.join(); b.join(); }\n")
    if subprocess.run(["g++", "-std=c++17", "-pthread", "-fsanitize=thread", str(src), "-o", str(exe)],
                      capture_output=True).returncode != 0:
        return False
    return "data race" in subprocess.run([str(exe)], capture_output=True, text=True).stderr


def test_team_reductions_are_ordered(tmp_path):
    """Every access to the team's shared state is ordered by a barrier: the
    slot set of a reduction is chosen by a counter that one thread advances in
    the same reduction."""
    if not sanitizer_runs(tmp_path):
        pytest.skip("ThreadSanitizer does not run here")
    exe = build(tmp_path, "team_threads.cpp", {"team.inc": ["common.cuh"]}, "-fsanitize=thread")
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and "data race" not in r.stderr, r.stdout + r.stderr[:4000]


# the reductions of the body in cluster_threads.cpp: 1 the mean, 2 the residual, then
# B, D, E of an iteration (3 4 5, 6 7 8, 9 10 11), 12 the true residual, ..., 22 the last mean
WAITS = [[0, 1], [2, 2], [0, 3], [2, 4], [0, 5], [2, 8], [1, 11], [0, 12], [2, 21], [0, 22], [1, 1, 2], [1, 7, 8]]


def test_cluster_leaves_together(tmp_path):
    """A CTA whose bounded wait ran out, in whichever reduction: all CTAs of the
    cluster leave behind the same barrier, and none posts into the shared
    memory of one that has left."""
    inc = {"cluster.inc": ["common.cuh", "cluster_team.cuh"]}
    runs = [(build(tmp_path, "cluster_threads.cpp", inc), [])]
    (tmp_path / "short").mkdir()
    short = build(tmp_path / "short", "cluster_threads.cpp", inc, "-DCUP2D_CLUSTER_POLLS=20")
    for exe, args in runs + [(short, w) for w in WAITS]:
        r = subprocess.run([str(exe), *map(str, args)], capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, (args, r.stdout, r.stderr)
