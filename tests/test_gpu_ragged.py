"""Transposition of 1- and 2-byte elements whose output rows start anywhere,
and of short rows staged as one range: the staged form and the form held in
shared memory, at the edges of their blocks and vectors."""
import pytest

torch = pytest.importorskip("torch")

from libmarshal_gb300 import lm

pytestmark = pytest.mark.gpu

STAGED, RESIDENT = 6, 7


def _check(T, a, B, e, method, offset=0):
    n = T * a * B * e
    g = torch.Generator(device="cuda").manual_seed(n + offset)
    raw = torch.randint(0, 256, (n + 64,), dtype=torch.uint8, device="cuda",
                        generator=g)
    before = raw.clone()
    dt = {1: torch.uint8, 2: torch.int16, 4: torch.int32, 8: torch.int64}[e]
    want = before[offset:offset + n].clone().view(dt).view(T, a, B) \
        .transpose(1, 2).reshape(-1).view(torch.uint8)
    lm.transpose_0100(raw.data_ptr() + offset, T, a, B, 1, method=method,
                      elem_bytes=e)
    torch.cuda.synchronize()
    assert torch.equal(raw[offset:offset + n], want)
    assert torch.equal(raw[:offset], before[:offset])
    assert torch.equal(raw[offset + n:], before[offset + n:])


# a (column lengths): around a vector, whole columns (up to 256 rows), the
# block heights 112, 120, 128, 240 and 248 and one row past each, several
# blocks with a last one of a few rows
ROWS = [2, 3, 15, 17, 31, 47, 113, 121, 129, 150, 225, 241, 249, 255, 257,
        260, 481, 487, 721, 1001]


@pytest.mark.parametrize("method", [STAGED, RESIDENT])
@pytest.mark.parametrize("e", [1, 2])
@pytest.mark.parametrize("a", ROWS)
def test_column_lengths(a, e, method):
    for B in (3, 15, 33, 190, 257, 1030):
        _check(1, a, B, e, method)


@pytest.mark.parametrize("e,offsets", [(1, range(16)), (2, range(0, 16, 2))])
def test_buffer_alignment(e, offsets):
    for off in offsets:
        for a, B in ((300, 205), (77, 304), (1024, 33), (40, 50)):
            _check(1, a, B, e, STAGED, off)
            _check(1, a, B, e, RESIDENT, off)


@pytest.mark.parametrize("e", [1, 2, 4, 8])
@pytest.mark.parametrize("B", [2, 3, 4, 5, 8, 9, 12, 16, 17, 30, 63, 64, 95, 119, 124,
                               191, 193])
def test_short_rows(B, e):
    """Rows staged as one range, and the widths just past it."""
    for T, a in ((1, 4099), (3, 1000), (2, 1537), (5, 257)):
        _check(T, a, B, e, STAGED)
        _check(T, a, B, e, RESIDENT)


@pytest.mark.parametrize("e", [1, 2])
def test_planner_large(e):
    """Past the form held in shared memory, through the planner's choice."""
    for T, a, B in ((1, 3000001, 15), (3, 1501, 9001), (1, 149, 300001)):
        _check(T, a, B, e, 0)


def test_near_the_limit():
    """Payloads that shared memory holds only without the extra rows."""
    for a, B in ((1001, 26816), (5007, 6001), (3001, 10007)):
        _check(1, a, B, 1, RESIDENT)


@pytest.mark.parametrize("e", [1, 2])
@pytest.mark.parametrize("groups", [1, 2, 3, 4, 6, 7, 8, 13, 14, 15, 28])
def test_groups_of_rows(groups, e):
    """Columns of so many 16-byte groups and a row less or more: groups are
    written seven (three) at a time with the rows of the one after."""
    for a in (groups * 16 // e - 1, groups * 16 // e + 1):
        for B in (7, 131, 517):
            _check(2, a, B, e, STAGED)
            _check(2, a, B, e, RESIDENT)


@pytest.mark.parametrize("a,B", [(905, 1082), (323, 1243), (2111, 853),
                                 (1217, 1213), (3301, 2503), (150, 9001)])
@pytest.mark.parametrize("off", [0, 3, 8])
def test_bytes_held_in_smaller_blocks(a, B, off):
    """Ragged blocks of bytes of each size that the held form chooses among."""
    n = a * B
    raw = torch.randint(0, 256, (n + 64,), dtype=torch.uint8, device="cuda")
    before = raw.clone()
    lm.transpose_0100(raw.data_ptr() + off, 1, a, B, 1, method=7, elem_bytes=1)
    torch.cuda.synchronize()
    assert torch.equal(raw[off:off + n],
                       before[off:off + n].view(a, B).t().reshape(-1))
    assert torch.equal(raw[:off], before[:off])
    assert torch.equal(raw[off + n:], before[off + n:])
