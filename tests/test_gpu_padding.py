"""Row padding and unpadding by tasks of byte ranges (lm_pad.cu), at the edges
of tasks, rows and vectors and on buffers at every alignment."""
import pytest

torch = pytest.importorskip("torch")

from libmarshal_gb300 import lm

pytestmark = pytest.mark.gpu

DT = {1: torch.uint8, 2: torch.int16, 4: torch.int32, 8: torch.int64}


def _check(e, x, y, pad, offset=0):
    n = y * pad * e
    g = torch.Generator(device="cuda").manual_seed(n + x + offset)
    raw = torch.randint(1, 256, (n + 64,), dtype=torch.uint8, device="cuda",
                        generator=g)
    before = raw.clone()
    data = before[offset:offset + n].clone().view(DT[e])
    ptr = raw.data_ptr() + offset
    want = torch.zeros_like(data)
    want.view(y, pad)[:, :x] = data[:y * x].view(y, x)
    lm.padding(ptr, x, y, pad, elem_bytes=e)
    assert torch.equal(raw[offset:offset + n], want.view(torch.uint8))
    data = torch.randint(1, 100, (y * pad,), device="cuda", generator=g).to(DT[e])
    raw[offset:offset + n] = data.view(torch.uint8)
    want.zero_()
    want[:y * x] = data.view(y, pad)[:, :x].reshape(-1)
    lm.unpadding(ptr, x, y, pad, elem_bytes=e)
    assert torch.equal(raw[offset:offset + n], want.view(torch.uint8))
    assert torch.equal(raw[:offset], before[:offset])
    assert torch.equal(raw[offset + n:], before[offset + n:])


@pytest.mark.parametrize("e", [1, 2, 4, 8])
def test_shapes(e):
    for x, y, pad in ((1, 1, 2), (0, 7, 5), (3, 100, 4), (15, 70, 16),
                      (16, 4000, 17), (1, 3000, 129), (17, 2049, 32),
                      (2047, 33, 2048), (2049, 33, 3000), (1024, 600, 1200),
                      (33000, 5, 33001), (5000, 101, 40000), (100003, 9, 100016),
                      (661, 16, 672), (4, 100000, 5)):
        _check(e, x, y, pad)


@pytest.mark.parametrize("e", [1, 2, 4, 8])
def test_alignments(e):
    for off in range(0, 16, e):
        for x, y, pad in ((37, 501, 40), (3001, 21, 3100), (2000, 61, 2500)):
            _check(e, x, y, pad, off)


@pytest.mark.parametrize("e,x,y,pad", [(4, 12289, 1024, 12320),
                                       (1, 30484, 2000, 30496),
                                       (2, 663, 50001, 672), (8, 25, 200000, 28)])
def test_large(e, x, y, pad):
    _check(e, x, y, pad)


@pytest.mark.parametrize("e", [1, 2, 4, 8])
@pytest.mark.parametrize("row", [15, 16, 17, 31, 32, 33])
def test_rows_about_a_vector(e, row):
    """Rows of one to two output vectors: a vector holds the end of one row
    and the whole or the start of the next."""
    for x in sorted({1, 7, row // 2, row - 1}):
        _check(e, x, 700, row)
        _check(e, x, 700, row, offset=16 - e)


@pytest.mark.parametrize("off", [0, 4, 12])
def test_calls_after_an_empty_one(off):
    """A call that starts no kernel books no tickets on the flags that are kept
    between calls."""
    raw = torch.zeros(4096, dtype=torch.uint8, device="cuda")
    for unpad in (0, 1):
        _check(4, 1000, 600, 1010, off)
        for x, y, pad in ((3, 0, 5), (0, 7, 0)):
            assert lm.lib().lm_debug_pad_stall(None, raw.data_ptr() + off, 4, x,
                                               y, pad, unpad, 0,
                                               1_000_000) is False
        _check(4, 1000, 600, 1010, off)


@pytest.mark.parametrize("x,pad", [(0, 1), (1, 2), (1, 3), (2, 3), (3, 4),
                                   (4, 5), (5, 9), (12, 14), (25, 26)])
def test_short_rows_of_doubles(x, pad):
    """A vector's two elements in one row, in two, or in a row's padding, over
    many tasks and on both halves of a vector."""
    for off in (0, 8):
        for y in (1, 7, 40001):
            _check(8, x, y, pad, off)
