"""The MatrixMarket size line as the Python wrapper reads it to size its buffers: a line it cannot
use is left to the parser, which names the error (the header is judged on the host: no GPU)."""
import pytest

from sparkx_b200 import build
import sparkx_b200.pkt as P

HEAD = b"%%MatrixMarket matrix coordinate pattern symmetric\n"


@pytest.fixture(scope="module", autouse=True)
def _lib():
    build.build_engine()


@pytest.mark.parametrize("size,want", [
    (b"3 3 1", (3, 1)), (b" 3\t3  1 ", (3, 1)), (b"3 4 1", (0, 0)), (b"3 3", (0, 0)), (b"3 3 99", (0, 0)),
    (b"+3 3 1", (0, 0)), (b"x 3 1", (0, 0)), (b"0" * 17 + b"003 3 1", (3, 1)),
    (b"9" * 20 + b" 3 1", (0, 0)), (b"1" * 5000 + b" 3 1", (0, 0)), (b"3 3 " + b"1" * 5000, (0, 0)),
], ids=lambda x: x[:12].decode() + f"_{len(x)}" if isinstance(x, bytes) else "")
def test_declared_size(size, want):
    assert P._mtx_declared(HEAD + b"% a comment\n\n" + size + b"\n1 2\n") == want


@pytest.mark.parametrize("size", [b"1" * 5000 + b" 3 1", b"3 3 " + b"9" * 4301, b"9" * 21 + b" 3 1", b"3 3 x", b"3 4 1"],
                         ids=lambda x: x[:12].decode() + f"_{len(x)}")
def test_the_parser_names_the_error(size):
    with pytest.raises(P.PktError) as e:
        P.mtx_to_csr(HEAD + size + b"\n1 2\n")
    assert e.value.status == P.E_PARSE
