"""The scalars that the batched Lanczos kernel's CTAs leave for each other.

Between two grid barriers the CTAs run in any order, so a word that one CTA
writes and another reads must have a barrier between the two accesses, for
every sequence of projecting and plain steps.  The kernel's accesses are laid
out here in barrier intervals, with the word numbers of batch_words.hpp
(compiled on the host).
"""
import ctypes
import itertools
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "nssdmrg_gb300" / "csrc"


@pytest.fixture(scope="module")
def words(tmp_path_factory):
    d = tmp_path_factory.mktemp("words")
    (d / "w.cpp").write_text('#include "batch_words.hpp"\n'
                             'extern "C" int owed(int step) { return nss::owed_word(step); }\n'
                             'extern "C" int alpha() { return nss::ST_ALPHA; }\n'
                             'extern "C" int hj() { return nss::ST_HJ; }\n'
                             'extern "C" int count() { return nss::ST_WORDS; }\n')
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", f"-I{CSRC}", "-o", str(d / "w.so"), str(d / "w.cpp")],
                   check=True)
    return ctypes.CDLL(str(d / "w.so"))


def accesses(words, rounds):
    """[(interval, 'w' or 'r', word, value)] of one solve, rounds[k] projections in step k.
    Writes are its first CTA's, reads every CTA's."""
    t, out = 0, []
    for k, r in enumerate(rounds):
        t += 1                                           # barrier behind the products
        out += [(t, "w", words.alpha(), k), (t, "w", words.hj(), k)]
        t += 1                                           # barrier behind the three-term step
        out.append((t, "r", words.alpha(), k))
        if k > 0:
            out.append((t, "r", words.owed(k - 1), k - 1))
        for _ in range(r):
            t += 1                                       # barrier behind the dots
            out.append((t, "w", words.hj(), k))
            t += 1                                       # barrier behind the update
            out += [(t, "r", words.alpha(), k), (t, "r", words.hj(), k)]
        out.append((t, "w", words.owed(k), k))
    return out


@pytest.mark.parametrize("steps", [1, 2, 4, 7])
def test_a_barrier_lies_between_write_and_read(words, steps):
    for rounds in itertools.product(range(3), repeat=min(steps, 5)):
        rounds = (rounds * 2)[:steps]
        acc = accesses(words, rounds)
        writes = [(t, w, v) for t, kind, w, v in acc if kind == "w"]
        for t, kind, word, value in acc:
            assert 0 <= word < words.count()
            if kind == "r":
                same = [x for x in writes if x[1] == word]
                assert all(x[0] != t for x in same), (rounds, "written and read between the same barriers", word, t)
                assert max(x for x in same if x[0] < t)[2] == value, (rounds, "an older value is read", word)
