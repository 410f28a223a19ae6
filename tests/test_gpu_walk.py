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
