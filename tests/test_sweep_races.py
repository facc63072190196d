"""The multigrid's smoothing kernels compiled for the CPU, one thread per CUDA
thread, under ThreadSanitizer: no access to shared or global memory is left
unordered by the kernels' own barriers, and what they compute is the two colour
passes to the bit.

The kernels' text is taken from the sources as it is; only the inline PTX of the
asynchronous copies and the __shared__ declarations are replaced
(cuda_on_host.h)."""
import os
import re
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "paris-git_b200", "csrc")

# id: configurations of k_rb_sweep_col (type, chunks of a staged row, rows, planes ahead, blocks per SM)
CONFIGS = [("float", 0, "16, 6, 3, 4"), ("float", 1, "16, 10, 2, 3"), ("float", 2, "48, 5, 1, 2"),
           ("double", 3, "16, 6, 2, 4"), ("double", 4, "16, 10, 2, 3")]


def between(text, start, end):
    a = text.index(start)
    return text[a:text.index(end, a)]


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    if not shutil.which("g++"):
        pytest.skip("no g++")
    read = lambda f: open(os.path.join(CSRC, f)).read()
    fast, sweep, col, common, ctx = (read(f) for f in ("mg_fast.cu", "mg_sweep.cuh", "mg_sweep_col.cuh", "common.cuh",
                                                       "ctx.cuh"))
    col = col[:col.index("// 16 bytes, asynchronously")] + col[col.index("// a configuration:"):]
    text = "\n".join([
        between(common, "// Boundary description", "// The inflow of a 'jet'"),
        "inline long cidx(int n0, int n1, int i, int j, int k) { return i + (long)n0 * (j + (long)n1 * k); }",
        "template <int BLOCK> double block_sum(double v, double*) { abort(); return v; }",
        between(fast, "static constexpr long kCoarseCells", "static inline dim3 row_grid"),
        between(sweep, "// wrap a coordinate into", "__device__ inline int sw_next"),
        between(ctx, "struct SwColGeo", "// One level of the B200 multigrid"),
        col,
        between(fast, "// t / d for 0 <= t", "// shared memory of k_coarse_cycle_smem"),
    ])
    text = text.replace("#pragma once", "")
    text = re.sub(r"extern __shared__ .*?unsigned char (\w+)\[\];", r"static unsigned char* const \1 = shared_raw;", text)
    text = text.replace("__shared__", "static")
    d = tmp_path_factory.mktemp("host")
    src, exe = str(d / "sweep.cpp"), str(d / "sweep")
    with open(src, "w") as f:
        f.write('#include "cuda_on_host.h"\n#include <string>\n' + text + "\n"
                + open(os.path.join(HERE, "sweep_on_host.cpp")).read())
    cols = " ".join(f"COL({t}, {q}, {c})" for t, q, c in CONFIGS)
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-ffp-contract=off", "-fsanitize=thread", "-w", "-I", HERE,
                        f"-DCOLUMN_CONFIGURATIONS={cols}", src, "-o", exe, "-lpthread"], capture_output=True, text=True)
    if "cannot find -ltsan" in r.stderr or "libtsan" in r.stderr:
        pytest.skip("no ThreadSanitizer")
    assert r.returncode == 0, r.stderr[-4000:]
    return exe


def run(program, *args):
    env = dict(os.environ, TSAN_OPTIONS="halt_on_error=1 exitcode=66")
    r = subprocess.run([program, *[str(a) for a in args]], capture_output=True, text=True, env=env, timeout=600)
    if "FATAL: ThreadSanitizer" in r.stderr:   # (its memory layout does not fit this kernel's)
        pytest.skip("ThreadSanitizer does not run here")
    assert r.returncode == 0, (r.returncode, r.stdout[-2000:], r.stderr[-3000:])


# whole rows, idle lanes, rows cut into tiles with a partial last one, a last
# row tile of two and of four rows, chunks of planes with a partial last one
@pytest.mark.parametrize("form", [0, 1, 2])
@pytest.mark.parametrize("cfg,n,per,zc", [
    (0, (20, 8, 6), (0, 1, 0), 4), (0, (64, 10, 6), (1, 0, 1), 4), (1, (72, 12, 4), (1, 1, 1), 2),
    (1, (120, 10, 4), (0, 0, 0), 4), (2, (136, 6, 4), (0, 1, 1), 4),
    (3, (32, 8, 6), (1, 1, 1), 4), (3, (20, 8, 6), (0, 0, 1), 2), (4, (60, 12, 4), (1, 0, 0), 4)])
def test_column_sweep(program, cfg, n, per, zc, form):
    run(program, "col", CONFIGS[cfg][0], cfg, *n, *per, form, zc)


# coarsest levels: odd extents over periodic seams (one, two, three axes), in a
# block and in one warp, and the levels above them
@pytest.mark.parametrize("ftype", ["float", "double"])
@pytest.mark.parametrize("nl,n,per", [(1, (5, 4, 7), (1, 1, 0)), (1, (3, 9, 5), (1, 1, 1)), (1, (3, 3, 5), (1, 1, 1)),
                                      (1, (6, 5, 4), (0, 1, 1)), (1, (5, 7, 3), (0, 0, 0)), (2, (6, 10, 6), (1, 1, 1))])
def test_coarse_cycle(program, nl, n, per, ftype):
    """One level: also the 32 passes cell after cell, to the bit."""
    run(program, "coarse", ftype, nl, *n, *per, 64)


@pytest.mark.parametrize("n,per", [((5, 7, 9), (1, 1, 1)), ((9, 4, 5), (1, 0, 1)), ((6, 5, 8), (1, 1, 1))])
def test_colour_passes(program, n, per):
    run(program, "passes", "double", 0, *n, *per)
