"""Segment walks (lm_walk.cu): 0100 on units of whole lines whose cycles are
longer than the whole-cycle form takes, through the public entry point."""
import pytest

torch = pytest.importorskip("torch")

from libmarshal_gb300 import lm

pytestmark = pytest.mark.gpu


def _convert(T, a, B, unit, e, graph=False):
    """(kernels launched, converted buffer, expected) of one in-place call."""
    n = T * a * B * unit
    g = torch.Generator(device="cuda").manual_seed(n)
    buf = torch.empty(n // 4, dtype=torch.int32, device="cuda")
    buf.random_(generator=g)
    want = buf.view(T, a, B, unit // 4).transpose(1, 2).reshape(-1)
    call = lambda: lm.transpose_0100(buf, T, a, B, unit // e, elem_bytes=e)
    if graph:
        gr = torch.cuda.CUDAGraph()
        with torch.cuda.graph(gr):
            call()
        gr.replay()
        torch.cuda.synchronize()
        return None, buf, want
    lm.prof_collect()
    lm.prof_enable(True)
    call()
    torch.cuda.synchronize()
    lm.prof_enable(False)
    return set(lm.prof_collect()), buf, want


# lanes per unit: 8, 12, 13, 32, 17 twice (two slices), 27 of 5 slices with a
# shorter last one; several tiles; a last block of positions without a start;
# cycles of 42 and 33 positions, some of which hold no start
SHAPES = [
    (1, 24, 5501, 128, 4), (1, 5501, 24, 192, 8), (1, 23, 5003, 208, 8),
    (1, 24, 1501, 512, 4), (1, 1501, 24, 528, 4), (1, 24, 503, 2096, 8),
    (3, 72, 100, 800, 8), (5, 33, 801, 128, 1), (2, 211, 401, 128, 4),
    (1, 128, 1024 * 64, 128, 4), (1, 2, 70001, 128, 2),
]


@pytest.mark.parametrize("shape", SHAPES)
def test_walk(shape, monkeypatch):
    monkeypatch.setenv("LM_NO_RESIDENT", "1")
    T, a, B, unit, e = shape
    ran, got, want = _convert(*shape)
    if T * a * B * unit >= 16 << 20 and _order(a, a * B - 1) > 32:
        assert {"walk_save", "walk"} <= ran
    assert torch.equal(got, want)


def _order(a, m):
    x, k = a % m, 1
    while x != 1 and k < 100:
        x, k = x * a % m, k + 1
    return k


def test_walk_short_cycles(monkeypatch):
    """Shapes whose cycles all have 33 to 99 positions: many hold no start."""
    monkeypatch.setenv("LM_NO_RESIDENT", "1")
    shapes = [(a, B) for a in range(30, 60) for B in range(2800, 2830)
              if 32 < _order(a, a * B - 1) < 99][:4]
    assert shapes
    for a, B in shapes:
        ran, got, want = _convert(1, a, B, 256, 4)
        assert {"walk_save", "walk"} <= ran
        assert torch.equal(got, want)


def test_walk_under_capture():
    """A captured call finds its cycles itself (no list is kept for it)."""
    lm.transpose_100(torch.zeros(1000 * 777, dtype=torch.int32, device="cuda"),
                     1000, 777, 1)  # the library's first call allocates
    _, got, want = _convert(1, 24, 11003, 128, 4, graph=True)
    assert torch.equal(got, want)


def test_walk_concurrent_streams():
    """Calls on several streams share one list and no scratch."""
    streams = [torch.cuda.Stream() for _ in range(4)]
    bufs = [torch.randint(-1000, 1000, (25 * 11001 * 32,), dtype=torch.int32,
                          device="cuda") for _ in streams]
    want = [b.view(25, 11001, 32).transpose(0, 1).reshape(-1) for b in bufs]
    torch.cuda.synchronize()
    for _ in range(3):
        for s, b in zip(streams, bufs):
            lm.transpose_100(b, 25, 11001, 32, stream=s)
            lm.transpose_100(b, 11001, 25, 32, stream=s)
    for s, b in zip(streams, bufs):
        lm.transpose_100(b, 25, 11001, 32, stream=s)
    torch.cuda.synchronize()
    for b, w in zip(bufs, want):
        assert torch.equal(b, w)


def test_walks_leave_room_for_the_lists_of_cycles(monkeypatch):
    """Shapes that are walked in segments do not take the room of the lists of
    whole cycles: after many of them a new shape's list is still kept."""
    monkeypatch.setenv("LM_NO_RESIDENT", "1")
    lm.lib().lm_marshal_finalize()
    for B in range(5501, 5521):  # 17 MB of 128-byte units each
        x = torch.zeros(24 * B * 32, dtype=torch.int32, device="cuda")
        lm.transpose_100(x, 24, B, 32)
    x = torch.arange(12 * 12 * 65536, dtype=torch.int32, device="cuda")
    want = x.view(12, 12, 65536).transpose(0, 1).reshape(-1)
    ran = []
    for _ in range(3):
        lm.prof_collect()
        lm.prof_enable(True)
        lm.transpose_100(x, 12, 12, 65536)
        torch.cuda.synchronize()
        lm.prof_enable(False)
        ran.append(set(lm.prof_collect()))
    assert ran == [{"cycle_leaders", "cycle_move"}, {"cycle_move"},
                   {"cycle_move"}]
    assert torch.equal(x, want)


def test_a_kept_list_takes_no_scratch():
    """A call on a shape whose list of cycles is kept allocates its walk's
    scratch, an eighth of the payload, and no memory for the list."""
    import ctypes
    cu = ctypes.CDLL("libcuda.so.1")
    pool, v = ctypes.c_void_p(), ctypes.c_uint64()
    torch.zeros(1, device="cuda")
    assert cu.cuDeviceGetDefaultMemPool(ctypes.byref(pool), 0) == 0

    def used(attr):  # 7: used now, 8: most since the last reset
        assert cu.cuMemPoolGetAttribute(pool, attr, ctypes.byref(v)) == 0
        return v.value

    a, B, words = 25, 30011, 32  # 96 MB of 128-byte units
    x = torch.zeros(a * B * words, dtype=torch.int32, device="cuda")
    for _ in range(2):
        lm.transpose_100(x, a, B, words)
    torch.cuda.synchronize()
    before = used(7)
    zero = ctypes.c_uint64(0)
    assert cu.cuMemPoolSetAttribute(pool, 8, ctypes.byref(zero)) == 0
    lm.transpose_100(x, a, B, words)
    torch.cuda.synchronize()
    walk = x.numel() * 4 // 8 + 2048
    assert used(8) - before < walk + (1 << 19)  # (the list: 1.5 MB)


def _ran(ptr, T, a, B, unit):
    lm.prof_collect()
    lm.prof_enable(True)
    lm.transpose_0100(ptr, T, a, B, unit // 8, elem_bytes=8)
    torch.cuda.synchronize()
    lm.prof_enable(False)
    return set(lm.prof_collect())


WALK, WAVE = {"walk_save", "walk"}, {"suffix_copy", "wave"}


# units on lines, halves of lines, sectors and off them; lanes that fill little
# of a warp (17 of 32), slices of a unit; below the size of L2 and with many
# tiles nothing but the alignment to 16 bytes counts
@pytest.mark.parametrize("T,a,mb,unit,off,ran", [
    (1, 24, 140, 128, 0, WALK), (1, 24, 140, 128, 64, WAVE),
    (1, 24, 140, 128, 16, WAVE), (1, 24, 110, 128, 64, WALK),
    (1, 24, 140, 192, 64, WALK), (1, 24, 140, 192, 32, WAVE),
    (1, 24, 140, 208, 0, WAVE), (1, 24, 110, 208, 0, WALK),
    (1, 24, 140, 272, 0, WAVE), (1, 24, 140, 320, 32, WALK),
    (1, 24, 140, 320, 16, WAVE), (1, 24, 140, 352, 16, WALK),
    (1, 24, 140, 528, 0, WAVE), (1, 24, 140, 640, 0, WALK),
    (2, 100, 280, 128, 32, WAVE), (12, 24, 280, 128, 32, WALK),
    (1, 24, 140, 1040, 48, WALK),
])
def test_walk_by_alignment(T, a, mb, unit, off, ran):
    B = (mb << 20) // (T * a * unit)
    n = T * a * B * unit
    raw = torch.randint(0, 256, (n + 256,), dtype=torch.uint8, device="cuda")
    before = raw.clone()
    first = _ran(raw.data_ptr() + off, T, a, B, unit)
    assert first - {"walk_leaders"} == ran
    want = before[off:off + n].view(T, a, B, unit).transpose(1, 2).reshape(-1)
    assert torch.equal(raw[off:off + n], want)
    assert torch.equal(raw[:off], before[:off])
    assert torch.equal(raw[off + n:], before[off + n:])


def test_walk_whose_list_is_not_kept(monkeypatch):
    """Under capture, and where no more lists are kept, each call finds its
    cycles: worth it from 80 MB on alone."""
    monkeypatch.setenv("LM_NO_RESIDENT", "1")
    lm.lib().lm_marshal_finalize()
    buf = torch.zeros(100 << 20, dtype=torch.uint8, device="cuda")
    shapes = [B for B in range(5501, 5601) if _order(24, 24 * B - 1) > 32][:64]
    for B in shapes:  # 17 MB each
        assert _ran(buf.data_ptr(), 1, 24, B, 128) == WALK | {"walk_leaders"}
    assert _ran(buf.data_ptr(), 1, 24, shapes[0], 128) == WALK
    staged = _ran(buf.data_ptr(), 1, 24, 20011, 128)  # 61 MB
    assert "staged_gather" in staged
    assert _ran(buf.data_ptr(), 1, 24, 30011, 128) == WALK | {"walk_leaders"}
    lm.lib().lm_marshal_finalize()
    assert _ran(buf.data_ptr(), 1, 24, 20011, 128) == WALK | {"walk_leaders"}
    lm.transpose_100(torch.zeros(1000 * 777, dtype=torch.int32, device="cuda"),
                     1000, 777, 1)
    for B in (20011, 30011):
        x = torch.arange(24 * B * 32, dtype=torch.int32, device="cuda")
        want = x.view(24, B, 32).transpose(0, 1).reshape(-1)
        gr = torch.cuda.CUDAGraph()
        with torch.cuda.graph(gr):
            lm.transpose_100(x, 24, B, 32)
        gr.replay()
        torch.cuda.synchronize()
        assert torch.equal(x, want)
