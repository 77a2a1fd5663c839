"""The rules that choose a call's kernel, compiled for the host: what they accept
stays within what the chosen kernel's index arithmetic holds."""
import os
import shutil
import subprocess

import pytest

from dawgs_gb300 import build

pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")


def run(tmp_path, body):
    """The words that a program printing `body`'s results writes."""
    src, exe = tmp_path / "rules.cpp", tmp_path / "rules"
    src.write_text('#include <cstdio>\n#include "ogs_internal.hpp"\nusing namespace ogsgb;\n'
                   "void out(long long x) { std::printf(\"%lld \", x); }\nint main() {\n" + body + "\n}\n")
    cuda = os.path.dirname(os.path.dirname(build.nvcc()))
    r = subprocess.run(["g++", "-std=c++17", "-I", build.INCLUDE, "-I", build.CSRC, "-I",
                        os.path.join(cuda, "include"), str(src), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return [int(x) for x in subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split()]


KS = [1, 2, 8, 9, 64, 1000, 2**26, 2**26 + 1, 2**27, 2**27 + 1, 2**31 - 1]


def test_scatter_in_node_order_takes_few_components(tmp_path):
    """A warp walks every component of its nodes, so large k goes to the tiles;
    no accepted k brings a component's place in a word near 32 bits."""
    body = "DevMaps m{}; m.nodes.nwords = 40; m.nodes.scatter = 1; FieldArgs f{}; Pattern p{0, 0, 0};\n"
    ks = KS + [16, 17]
    body += "".join(f"f.K = {k}; out(scatter_applies(m, f, p, 8)); out(scatter_applies(m, f, p, 4));\n" for k in ks)
    got = run(tmp_path, body)
    assert got[::2] == [int(k <= 8) for k in ks] and got[1::2] == [int(k <= 16) for k in ks]


def test_scatter_in_node_order_takes_handles_with_most_nodes_in_rows(tmp_path):
    """Its time goes with all nodes, that of the column lists with those in rows."""
    body = "ogs_handle_s h; h.N = 1000;\n"
    body += "".join(f"h.nnzT = {n}; out(scatter_share(&h));\n" for n in (1, 500, 749, 750, 1000))
    assert run(tmp_path, body) == [0, 0, 0, 1, 1]


def test_lone_vectors_end_with_the_field(tmp_path):
    """The last vectors of lone tiles, of the largest mesh too: none that reaches
    past the last node is taken whole."""
    cases = [(0, 0, 4, 4), (0, 0, 4, 3), (256, 252, 4, 512), (256, 252, 4, 511), (256, 254, 2, 511),
             (2**31 - 256, 252, 4, 2**31 - 1), (2**31 - 256, 248, 4, 2**31 - 1), (2**31 - 256, 254, 2, 2**31 - 1),
             (2**31 - 256, 254, 1, 2**31 - 1), (2**31 - 256, 255, 1, 2**31 - 1)]
    got = run(tmp_path, "".join(f"out(lone_vector_in({b}, {at}, {v}, {n}));\n" for b, at, v, n in cases))
    assert got == [int(b + at + v <= n) for b, at, v, n in cases]


def test_units_of_a_tile_fit_32_bits(tmp_path):
    """The largest k that the pipelines and wide tiles take keeps its last unit and
    its bytes below 2^32; separate arrays always do."""
    got = run(tmp_path, "".join(f"out(units_fit({k}, false)); out(units_fit({k}, true));\n" for k in KS))
    assert got[1::2] == [1] * len(KS)
    for k, fit in zip(KS, got[::2]):
        assert fit == int(32 * k - 1 < 2**32), k
        assert not fit or 8 * k < 2**32


def test_lone_tiles_by_the_field_and_the_share(tmp_path):
    """Handles with lone tiles: large fields, mostly lone nodes, and 8-byte folds
    that cost more or nothing."""
    body = "DevMaps m{}; m.nltiles = 3; m.nodes.nwords = 9;\n"
    cases = [(n, lone, b, c) for n in (1000, 4000000, 8000000) for lone in (0.56, 0.66) for b in (4, 8) for c in (0, 1)]
    for n, lone, b, c in cases:
        body += f"m.b[1].nnodes = {n}; m.b[1].n = {int(n * lone)}; out(lone_folds(m, {b}, {c})); out(lone_gathers(m, {b}));\n"
    body += "m.nodes.nwords = 0; out(lone_gathers(m, 8)); m.nltiles = 0; out(lone_folds(m, 8, true));\n"
    got = run(tmp_path, body)
    for (n, lone, b, c), f, g in zip(cases, got[::2], got[1::2]):
        large = n * b >= 30 * 2**20
        assert g == int(large), (n, lone, b, c)
        assert f == int(large or lone >= 0.65 or (c and b == 8)), (n, lone, b, c)
    assert got[-2:] == [0, 0]
