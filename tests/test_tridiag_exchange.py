"""Exchange of the register-resident tridiagonalisation (csrc/tridiag_exchange.cuh,
compiled for the host): on the barrier of the partial sums every CTA of a cluster
waits for a word of every CTA, its only order against their barriers of the step
before, and for exactly the words that are sent to it."""
import ctypes
import pathlib
import shutil
import subprocess

import pytest

CSRC = pathlib.Path(__file__).resolve().parents[1] / "atlasq_gb300" / "csrc"
WARPS = 8


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
        "int zeros(int C) { return exchange::zeros(C); }\n"
        "int dot_words(int q, int C) { return exchange::dot_words(q, C); }\n"
        "int dot_pitch(int C) { return exchange::dot_pitch(C); }\n"
        "}\n")
    subprocess.run([cxx, "-shared", "-fPIC", "-x", "c++", str(d / "x.cpp"), "-o", str(d / "x.so")], check=True)
    return ctypes.CDLL(str(d / "x.so"))


@pytest.mark.parametrize("C", range(2, 17))
def test_every_cta_waits_for_every_peer(rules, C):
    assert rules.zeros(C) <= WARPS  # a warp sends one
    for q in range(C):
        shares = [w for w in range(WARPS) if rules.dot_dest(w, C) == q]
        sent = len(shares) + (WARPS <= q < WARPS + rules.zeros(C))  # by each CTA, to CTA q
        assert sent == rules.dot_words(q, C) >= 1
        # where they land: the pitch keeps the senders apart, and all within 16 words
        places = [s * rules.dot_pitch(C) + w // C for s in range(C) for w in shares or [0]]
        assert len(set(places)) == C * sent and max(places) < 16
