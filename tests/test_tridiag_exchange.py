"""Exchange of the register-resident tridiagonalisation (csrc/tridiag_exchange.cuh):
in every step every CTA of a cluster waits, on the barrier of the partial sums, for
a word of every CTA (its only order against their barriers of the step before), and
for exactly the bytes that are sent to it.  The senders are restated from the
kernel's pass; the counts are the header's, compiled for the host."""
import ctypes
import pathlib
import shutil
import subprocess

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "atlasq_gb300" / "csrc"
WARPS, THREADS = 8, 256


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("exchange")
    (d / "x.cpp").write_text(
        f'#include "{CSRC / "tridiag_exchange.cuh"}"\n'
        'extern "C" {\n'
        "int dot_dest(int w, int C) { return exchange::dot_dest(w, C); }\n"
        "int zero_dest(int w, int C) { return exchange::zero_dest(w, C); }\n"
        "int slice(int n, int C, int t) { return exchange::slice(n, C, t); }\n"
        "int bytes1(int n, int C, int V, int t, int q, int j) { return exchange::bytes1(n, C, V, t, q, j); }\n"
        "}\n")
    subprocess.run([cxx, "-shared", "-fPIC", "-x", "c++", str(d / "x.cpp"), "-o", str(d / "x.so")], check=True)
    return ctypes.CDLL(str(d / "x.so"))


@pytest.mark.parametrize("n,C,cpt", [(129, 4, 2), (200, 3, 2), (256, 8, 2), (257, 16, 2), (300, 10, 2), (511, 10, 2),
                                     (512, 16, 2), (512, 9, 2), (513, 16, 4), (1023, 16, 4), (1024, 16, 4),
                                     (1024, 8, 4)])
def test_every_cta_waits_for_every_peer(rules, n, C, cpt):
    S = rules.slice(n, C, cpt)
    G = 1
    while G < 8 and cpt * (THREADS // (2 * G)) >= n:  # row groups of a CTA
        G *= 2
    V = C * G
    for j in sorted({0, 1, n // 3, n - n // C - 1, n - S, n - 3, n - 2}):
        for q in range(C):
            words = [0] * C  # dot words and zeros that reach CTA q, by sender
            for src in range(C):
                for w in range(WARPS):
                    words[src] += rules.dot_dest(w, C) == q
                    words[src] += rules.zero_dest(w, C) == q
            assert min(words) > 0, (j, q, words)
            # every thread whose columns are in use sends its cpt partial sums, one owner a row too
            cols = sum(1 for c0 in range(0, n, cpt) if c0 + cpt - 1 > j and c0 // S == q)
            assert rules.bytes1(n, C, V, cpt, q, j) == 4 * sum(words) + cols * (V + 1) * cpt * 8
