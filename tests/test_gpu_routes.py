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
    (15001, 2330, 3, 4, 0, True), (15001, 230, 3, 4, 0, True),
    (9001, 400, 3, 8, 0, False), (9001, 700, 3, 8, 0, True),
    (9001, 3000, 4, 4, 4, True), (9001, 3000, 4, 4, 0, False),  # vectors
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


@pytest.mark.parametrize("T,a,B,b,e,off,ran", [
    # units of one element: long tiles held, short ones and vector columns not
    (1, 41, 1598, 1, 1, 0, {"resident"}), (66, 363, 17, 1, 8, 0, {"bs_tile"}),
    (22, 246, 74, 1, 8, 0, {"resident"}), (62, 8, 8266, 1, 4, 0, {"bs_cluster"}),
    (1, 4, 17951, 1, 2, 0, {"bs_cluster"}),
    (2108, 2679, 2, 1, 2, 2, {"bs_tile"}),  # many tiles of many rows
    # units of several, written one element at a time either way
    (2, 92, 30, 45, 1, 0, {"resident"}), (148, 91, 2, 163, 1, 0, {"bs_tile"}),
    (35, 3, 2405, 86, 1, 1, {"bs_cluster"}),
    # clusters that do not fit at once
    (9, 327, 38, 105, 2, 0, {"resident"}), (14, 15, 27, 706, 4, 0, {"bs_cluster"}),
])
def test_held_or_tiles(T, a, B, b, e, off, ran):
    assert _route(T, a, B, b, e, off) == ran


def test_tiles_or_short_cycles():
    """Units whose cycles are short: whole cycles where their list is kept."""
    lm.lib().lm_marshal_finalize()
    assert _route(1, 4, 40, 768, 2) == {"bs_cluster"}
    for _ in range(2):
        ran = _route(21, 8, 2, 847, 8) - {"cycle_leaders"}
        assert ran == {"cycle_move"}


@pytest.mark.parametrize("T,a,b,e,off,square", [
    (1, 335, 31, 1, 0, False), (1, 1152, 31, 1, 0, False),
    (1, 280, 13, 1, 8, False), (1, 621, 9, 1, 0, True),
    (1, 3912, 7, 1, 0, False), (1, 2421, 15, 2, 2, False),
    (1, 1000, 13, 2, 0, True), (1, 335, 7, 4, 0, True), (3, 400, 3, 8, 8, True),
])
def test_squares_of_units(T, a, b, e, off, square):
    assert (_route(T, a, a, b, e, off) == {"square"}) == square


@pytest.mark.parametrize("a,B,off,held", [
    (11675, 2179, 0, False), (20854, 1455, 1, False), (3758, 7173, 0, False),
    (15048, 1907, 8, True),   # 8-byte vectors
    (13228, 1893, 0, True), (9148, 2673, 0, True), (4001, 4003, 1, True),
])
def test_bytes_near_the_limit_of_the_held_form(a, B, off, held):
    assert (_route(1, a, B, 1, 1, off) == {"resident"}) == held


@pytest.mark.parametrize("a,B,b,e", [(12684, 6629, 1, 1), (12700, 6629, 1, 1),
                                     (12684, 947, 7, 1), (25000, 600, 3, 2),
                                     (30100, 301, 9, 1)])
def test_first_call_of_a_stash_plan(a, B, b, e):
    """A plan that tries sizes beyond the limit of shared memory, in a thread
    that has planned nothing yet: neither its call nor the next one finds the
    refused size's error."""
    import threading
    n = a * B * b * e
    raw = torch.randint(0, 256, (n,), dtype=torch.uint8, device="cuda")
    want = raw.view(a, B, b * e).transpose(0, 1).reshape(-1)
    failed = []

    def work():
        for method, x in ((3, raw), (0, raw.clone())):
            try:
                lm.transpose_0100(x, 1, a, B, b, method=method, elem_bytes=e)
            except Exception as ex:  # noqa: BLE001
                failed.append((method, str(ex)))
        torch.cuda.synchronize()

    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert not failed
    assert torch.equal(raw, want)
