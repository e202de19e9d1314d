"""Kernel sequences (csrc/isf_seq.cu) against a CUDA runtime that records what
it is asked for (seq_host.cu, seq_runtime.cpp): no GPU."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "schroedingerssmoke.jl_b200")
CSRC = os.path.join(PKG, "csrc")


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    import __graft_entry__ as ge
    b = ge.load_builder()
    exe = str(tmp_path_factory.mktemp("seq") / "seq_host")
    cmd = [b.NVCC, *b.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-cudart", "none", "-I", b.INCLUDE, "-I", CSRC, "-o",
           exe, os.path.join(HERE, "seq_host.cu"), os.path.join(HERE, "seq_runtime.cpp"), os.path.join(CSRC, "isf_seq.cu")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def go(*args):
        r = subprocess.run([exe, *map(str, args)], capture_output=True, text=True, timeout=60)
        assert r.returncode == 0, (args, r.returncode, r.stdout, r.stderr)
        *lines, end = r.stdout.splitlines()
        assert end == "mode 0 graphs 0"   # capture mode as it was, no graph left
        return lines

    return go


def test_a_sequence_becomes_a_graph_with_each_call_s_arguments(run):
    plain = [f"launch {10 * c + k}" for c in (1, 2, 3) for k in range(3)]
    assert run("repeat", 6) == plain + [f"graph {c}0 {c}1 {c}2" for c in (4, 5, 6)]


@pytest.mark.parametrize("done", [0, 1, 2])
def test_kernels_before_a_failure_run(run, done):
    """A call that fails on the host after some of its kernels has launched
    those, as it does without recording."""
    assert run("stop", done) == [f"launch {10 + k}" for k in range(done)] + ["rc 1 stopped recording 0"]


@pytest.mark.parametrize("bad", [0, 1, 2])
def test_a_launch_that_fails_is_reported_by_its_pass(run, bad):
    done = [f"launch {10 + k}" for k in range(bad)]
    assert run("launch", bad) == done + [f"rc 2 pass {'abc'[bad]}"]


def test_no_host_memory_while_a_graph_is_built(run):
    """Whichever host allocation of the building call fails, the call reports
    it or launches its kernels, the thread's capture mode is as it was, and the
    next call launches its own three kernels once."""
    for n in range(100):
        lines = run("build", n)[9:]
        i = next(k for k, line in enumerate(lines) if line.startswith("rc "))
        assert lines[i] in ("rc 0 mode 0", "rc 3 mode 0"), (n, lines)
        kernels = lambda c: [[f"launch {10 * c + k}" for k in range(3)], [f"graph {c}0 {c}1 {c}2"]]  # noqa: E731
        assert lines[:i] in ([[]] if lines[i].startswith("rc 3") else kernels(4)), (n, lines)
        if lines[-1] == "all":
            break
        assert lines[i + 1:] in kernels(5), (n, lines)
    assert lines[-1] == "all" and n >= 5


def test_no_host_memory_for_the_recorded_launches(run):
    seen = []
    while not seen or seen[-1] != "all":
        (line,) = run("reserve", len(seen))
        seen.append(line)
    assert seen == ["no room"] * (len(seen) - 1) + ["all"] and len(seen) >= 4
