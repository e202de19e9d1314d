"""The (x, y) tiles of the kernels over cells (cell_tiles_host.cu): no GPU."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "schroedingerssmoke.jl_b200", "csrc")
LENS = (8, 12, 16, 20, 24, 32, 40, 48, 50, 56, 64, 80, 96, 100, 112, 128, 160, 192, 200, 256, 384, 512)


def up(n, m):
    return -(-n // m) * m


def test_every_cell_once_and_few_idle_lanes(tmp_path):
    import __graft_entry__ as ge
    b = ge.load_builder()
    exe = str(tmp_path / "cell_tiles")
    cmd = [b.NVCC, *b.ARCH, "-std=c++17", "--expt-relaxed-constexpr", "-I", b.INCLUDE, "-I", CSRC, "-o", exe,
           os.path.join(HERE, "cell_tiles_host.cu")]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    pairs = [(x, y) for x in LENS for y in LENS]
    r = subprocess.run([exe], input="\n".join(f"{x} {y}" for x, y in pairs), capture_output=True, text=True, timeout=60)
    out = [line.split() for line in r.stdout.splitlines()]
    assert len(out) == len(pairs)
    for (x, y), (ok, lanes) in zip(pairs, out):
        assert ok == "ok", (x, y)
        # within a third of the best of the three widths
        best = min(up(x, w) * up(y, 256 // w) for w in (8, 16, 32))
        assert 3 * int(lanes) < 4 * best or int(lanes) == best, (x, y, lanes, best)
