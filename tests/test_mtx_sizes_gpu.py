"""MatrixMarket texts whose size line declares another number of entries than they
hold, against the oracle's parser."""
import numpy as np
import pytest

from oracle import oracle as O
import sparkx_b200.pkt as P

pytestmark = pytest.mark.gpu


def test_size_lines_that_declare_too_few_too_many_or_nothing():
    """The result does not depend on the size line's entry count: it only sizes the buffers."""
    body = "".join(f"{i} {j}\n" for i, j in ((1, 2), (3, 2), (4, 4), (5, 1), (2, 1)))
    head = "%%MatrixMarket matrix coordinate pattern {}\n% note\n\n5 5 {}\n"
    for kind in ("symmetric", "general"):
        want = O.mtx_to_csr((head.format(kind, 5) + body).encode())
        for nnz in (0, 1, 4, 5, 6, 100000):
            off, nbr = P.mtx_to_csr((head.format(kind, nnz) + body).encode())
            assert np.array_equal(off, want[0]) and np.array_equal(nbr, want[1]), (kind, nnz)
