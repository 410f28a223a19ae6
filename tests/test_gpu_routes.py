"""Which form takes a conversion where two of them are close or far apart, by
the kernels that ran, and that the result is right either way."""
import pytest

torch = pytest.importorskip("torch")

from libmarshal_gb300 import lm

pytestmark = pytest.mark.gpu

STASH = {"stash_save", "stash_wave"}
WAVE = {"suffix_copy", "wave"}


def _route(T, a, B, b, e, off=0):
    """The kernels of a 0100(T, a, B, b), checked against torch."""
    n = T * a * B * b * e
    raw = torch.randint(0, 256, (n + 64,), dtype=torch.uint8, device="cuda")
    before = raw.clone()
    lm.prof_collect()
    lm.prof_enable(True)
    lm.transpose_0100(raw.data_ptr() + off, T, a, B, b, elem_bytes=e)
    torch.cuda.synchronize()
    lm.prof_enable(False)
    ran = set(lm.prof_collect())
    want = before[off:off + n].view(T, a, B, b * e).transpose(1, 2).reshape(-1)
    assert torch.equal(raw[off:off + n], want)
    assert torch.equal(raw[:off], before[:off])
    assert torch.equal(raw[off + n:], before[off + n:])
    return ran


@pytest.mark.parametrize("a,B,b,e,off,stash", [
    (7400, 1214, 7, 1, 0, True), (15001, 3994, 7, 1, 1, True),
    (15001, 80, 33, 2, 0, True), (15001, 423, 33, 2, 2, True),
    (7400, 446, 127, 1, 0, True), (7000, 1214, 7, 1, 0, False),  # rows
    (15001, 420, 129, 1, 0, False),                    # units of 128 bytes
    (15001, 2330, 3, 4, 0, True), (15001, 600, 3, 4, 0, False),
    (30001, 600, 3, 8, 0, False),
    (28775, 4005, 1, 2, 0, True), (28775, 3995, 1, 2, 0, False),
])
def test_stash(a, B, b, e, off, stash):
    assert (_route(1, a, B, b, e, off) - {"stash_offsets"} == STASH) == stash


@pytest.mark.parametrize("a,mb,b,e,off,wave", [
    (1000, 180, 3, 4, 0, False), (1000, 230, 3, 4, 0, True),
    (1000, 230, 33, 2, 0, False), (1000, 270, 33, 2, 0, True),
    (1000, 150, 9, 1, 0, False), (1000, 170, 9, 1, 0, True),
    (1000, 130, 3, 8, 0, False), (1000, 160, 3, 8, 0, True),
    (1000, 100, 2, 8, 0, True), (1000, 120, 2, 8, 8, False),  # whole vectors
    (100, 270, 21, 2, 0, True), (97, 230, 11, 4, 4, True),    # even heights
])
def test_wave_of_units_of_elements(a, mb, b, e, off, wave):
    B = (mb << 20) // (a * b * e)
    assert (_route(1, a, B, b, e, off) == WAVE) == wave
