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


BUILD_AT = 16   # the call of a sequence that builds its graph


def plain(c, kernels=(0, 1, 2)):
    return [f"launch {10 * c + k}" for k in kernels]


def graph(c, kernels=(0, 1, 2)):
    return ["graph " + " ".join(str(10 * c + k) for k in kernels)]


def calls(form, first, last, kernels=(0, 1, 2)):
    return [line for c in range(first, last + 1) for line in form(c, kernels)]


def test_a_sequence_becomes_a_graph_with_each_call_s_arguments(run):
    assert run("repeat", 20) == calls(plain, 1, 15) + calls(graph, 16, 20)


def test_a_handle_of_few_calls_builds_no_graph(run):
    """A graph costs what it saves on about fifteen calls."""
    assert run("repeat", 15) == calls(plain, 1, 15)


def test_large_grids_launch_their_kernels_as_they_come(run):
    assert run("large", 20) == calls(plain, 1, 20)


def test_another_sequence_of_the_same_call_has_a_graph_of_its_own(run):
    two = (0, 2)
    assert run("other", 18, 18) == (calls(plain, 1, 15) + calls(graph, 16, 18) + calls(plain, 19, 33, two) +
                                    calls(graph, 34, 36, two))


@pytest.mark.parametrize("before", [0, 17])
@pytest.mark.parametrize("done", [0, 1, 2])
def test_kernels_before_a_failure_run(run, done, before):
    """A call that fails on the host after some of its kernels has launched
    those, as it does without recording."""
    lines = run("stop", done, before)
    tail = [f"launch {10 * (before + 1) + k}" for k in range(done)] + ["rc 1 stopped recording 0"]
    assert lines[len(lines) - len(tail):] == tail and len(lines) == (45 + 2 if before else 0) + len(tail)


@pytest.mark.parametrize("before", [0, 17])
@pytest.mark.parametrize("bad", [0, 1, 2])
def test_a_launch_that_fails_is_reported_by_its_pass(run, bad, before):
    lines = run("launch", bad, before)
    tail = [f"launch {10 * (before + 1) + k}" for k in range(bad)] + [f"rc 2 pass {'abc'[bad]}"]
    assert lines[len(lines) - len(tail):] == tail and len(lines) == (45 + 2 if before else 0) + len(tail)


def test_no_host_memory_while_a_graph_is_built(run):
    """Whichever host allocation of the building call fails, the call reports
    it or launches its kernels, the thread's capture mode is as it was, and the
    next call launches its own three kernels once."""
    for n in range(100):
        lines = run("build", n, 15)[45:]
        i = next(k for k, line in enumerate(lines) if line.startswith("rc "))
        assert lines[i] in ("rc 0 mode 0", "rc 3 mode 0"), (n, lines)
        assert lines[:i] in ([[]] if lines[i].startswith("rc 3") else [plain(16), graph(16)]), (n, lines)
        if lines[-1] == "all":
            break
        assert lines[i + 1:] in (plain(17), graph(17)), (n, lines)
    assert lines[-1] == "all" and n >= 5


def test_no_host_memory_for_a_note(run):
    """A call that only notes its kernels does not fail for want of memory."""
    for n in range(10):
        lines = run("build", n)
        assert lines[:4] == plain(1) + ["rc 0 mode 0"] and lines[4:7] == plain(2), (n, lines)


def test_no_host_memory_for_the_recorded_launches(run):
    seen = []
    while not seen or seen[-1] != "all":
        (line,) = run("reserve", len(seen))
        seen.append(line)
    assert seen == ["no room"] * (len(seen) - 1) + ["all"] and len(seen) >= 4
