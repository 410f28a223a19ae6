"""Square transpositions by block pairs (k_square), through the planner."""
import pytest

torch = pytest.importorskip("torch")

from libmarshal_gb300 import lm

pytestmark = pytest.mark.gpu


def _check(T, a, b, e, offset=0):
    n = T * a * a * b * e
    g = torch.Generator(device="cuda").manual_seed(n + offset)
    raw = torch.randint(0, 256, (n + 64,), dtype=torch.uint8, device="cuda",
                        generator=g)
    before = raw.clone()
    want = before[offset:offset + n].view(T, a, a, b * e).transpose(1, 2) \
        .reshape(-1)
    lm.prof_collect()
    lm.prof_enable(True)
    lm.transpose_0100(raw.data_ptr() + offset, T, a, a, b, elem_bytes=e)
    torch.cuda.synchronize()
    lm.prof_enable(False)
    ran = set(lm.prof_collect())
    assert torch.equal(raw[offset:offset + n], want)
    assert torch.equal(raw[:offset], before[:offset])
    assert torch.equal(raw[offset + n:], before[offset + n:])
    return ran


# around one block, odd and even numbers of block rows, last blocks of a row
@pytest.mark.parametrize("e", [1, 2, 4, 8])
@pytest.mark.parametrize("a", [128, 129, 136, 140, 200, 255, 256,
                               257, 264, 333, 1000, 1016, 1118, 2056])
def test_sizes(a, e):
    ran = _check(1, a, 1, e)
    if a > 128 and (e >= 4 or a * e % 8 == 0):
        assert ran == {"square"}
    _check(3, a, 1, e)


@pytest.mark.parametrize("unit,e", [(6, 2), (8, 4), (12, 4), (16, 8), (20, 4),
                                    (24, 8), (32, 8), (3, 1)])
def test_units(unit, e):
    for a in (129, 200, 333):
        _check(2, a, unit // e, e)


@pytest.mark.parametrize("e", [1, 2, 4, 8])
def test_alignment(e):
    for off in range(0, 16, e):
        _check(1, 328, 1, e, off)
        _check(1, 177, 2, e, off)


def test_large():
    for a, e in ((5001, 4), (6000, 1), (4100, 2), (3001, 8)):
        assert _check(1, a, 1, e) == {"square"}


def test_under_capture():
    x = torch.randint(0, 1 << 30, (700, 700), dtype=torch.int32, device="cuda")
    want = x.t().contiguous()
    y = x.clone()
    lm.transpose_100(y, 700, 700, 1)  # the library's first call allocates
    gr = torch.cuda.CUDAGraph()
    with torch.cuda.graph(gr):
        lm.transpose_100(x, 700, 700, 1)
    gr.replay()
    torch.cuda.synchronize()
    assert torch.equal(x, want)
