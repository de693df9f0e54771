"""MatrixMarket bodies at the edges of their kernels: entry counts around the sort's
rounds of 1024 and blocks of 4096, vertex counts around each further bit and digit of
the keys, bodies that end anywhere in a 16-byte word, lines without entries, rows
that cross groups of 32; against the oracle's parser."""
import numpy as np
import pytest

from oracle import oracle as O
import sparkx_b200.pkt as P

pytestmark = pytest.mark.gpu


def _check(text):
    want = O.mtx_to_csr(text)
    off, nbr = P.mtx_to_csr(text)
    assert np.array_equal(off, want[0]) and np.array_equal(nbr, want[1])


def _text(n, i, j, kind, sep="\n", end="\n"):
    return ("%%MatrixMarket matrix coordinate pattern " + kind + f"\n{n} {n} {len(i)}\n" +
            sep.join(f"{a} {b}" for a, b in zip(i.tolist(), j.tolist())) + end).encode()


@pytest.mark.parametrize("n", [1, 2, 3, 16, 17, 256, 257, 65536, 65537, 1 << 20, 5_000_000])
@pytest.mark.parametrize("m", [0, 1, 31, 33, 1023, 1024, 1025, 4097, 20_000])
def test_entry_and_vertex_counts(n, m):
    rng = np.random.default_rng(n + m)
    i, j = rng.integers(1, n + 1, m), rng.integers(1, n + 1, m)  # any order, with repeats and loops
    _check(_text(n, i, j, "general"))
    _check(_text(n, np.maximum(i, j), np.minimum(i, j), "symmetric"))


@pytest.mark.parametrize("pad", range(17))
def test_body_lengths_and_empty_lines(pad):
    i, j = np.arange(2, 41), np.arange(1, 40)
    for sep in ("\n", "\r\n", "\n\n", "\n%x\n", " \n\t"):
        for end in ("", "\n", "\n\n", " " * pad, "\n" * pad, "\n%" + "y" * pad):
            _check(_text(40, i, j, "symmetric", sep, end))


@pytest.mark.parametrize("m", [40, 1000, 30_000])
def test_one_long_row(m):
    i = np.full(m, 7)
    _check(_text(50_000, i, np.random.default_rng(m).permutation(m) + 1, "general"))
