"""Large single transpositions and SoA <-> ASTA conversions in the ordered form
(k_wave), forward and backward, through the planner."""
import pytest

torch = pytest.importorskip("torch")

from libmarshal_gb300 import lm

pytestmark = pytest.mark.gpu


def _check(a, B, b, e, offset=0, wave=True):
    n = a * B * b * e
    g = torch.Generator(device="cuda").manual_seed(a + offset)
    raw = torch.randint(0, 256, (n + 64,), dtype=torch.uint8, device="cuda",
                        generator=g)
    before = raw.clone()
    want = before[offset:offset + n].view(a, B, b * e).transpose(0, 1) \
        .reshape(-1)
    lm.prof_collect()
    lm.prof_enable(True)
    lm.transpose_100(raw.data_ptr() + offset, a, B, b, elem_bytes=e)
    torch.cuda.synchronize()
    lm.prof_enable(False)
    ran = set(lm.prof_collect())
    assert torch.equal(raw[offset:offset + n], want)
    assert torch.equal(raw[:offset], before[:offset])
    assert torch.equal(raw[offset + n:], before[offset + n:])
    if wave:
        assert ran == {"wave", "suffix_copy"}


# output rows of whole vectors and not, both directions, last blocks of one
# row or column, whole rows (one block column) and whole columns
@pytest.mark.parametrize("a,B,b,e", [
    (20000, 8192, 1, 1), (16001, 16385, 1, 1), (1001, 268167, 1, 1),
    (268167, 1001, 1, 1), (149, 1500001, 1, 1), (16000001, 15, 1, 1),
    (12000, 8000, 1, 2), (12001, 8003, 1, 2), (20003, 5001, 1, 2),
    (3000001, 40, 1, 2), (18, 7000001, 1, 2),
    (9001, 6000, 1, 4), (6000, 9001, 1, 4), (12289, 8193, 1, 4),
    (1000001, 65, 1, 4), (106, 1178589, 1, 4), (5000001, 17, 1, 4),
    (11871, 6065, 1, 8), (6065, 11872, 1, 8), (779268, 80, 1, 8),
    (101, 125000, 8, 4), (125000, 101, 8, 4), (9001, 5003, 2, 8),
    (40000, 501, 3, 4), (501, 40000, 5, 4), (70001, 120, 6, 8),
])
def test_wave(a, B, b, e):
    _check(a, B, b, e)


@pytest.mark.parametrize("e", [1, 2, 4, 8])
def test_alignment(e):
    for off in {e, 16 - e, 8}:
        _check(8192 * 8 // e, 4100, 1, e, off)
        _check(2000001 // e, 160, 1, e, off, wave=False)


def test_under_capture():
    x = torch.randint(0, 1 << 30, (9001 * 6001,), dtype=torch.int32,
                      device="cuda")
    want = x.view(9001, 6001).t().reshape(-1)
    lm.transpose_100(x.clone(), 9001, 6001, 1)  # the first call allocates
    gr = torch.cuda.CUDAGraph()
    with torch.cuda.graph(gr):
        lm.transpose_100(x, 9001, 6001, 1)
    gr.replay()
    torch.cuda.synchronize()
    assert torch.equal(x, want)
    gr.replay()
    torch.cuda.synchronize()
    assert torch.equal(x, want.view(9001, 6001).t().reshape(-1))


def test_concurrent_streams():
    """Waves on several streams: every CTA's waits end whatever the others
    hold of the GPU."""
    streams = [torch.cuda.Stream() for _ in range(4)]
    bufs = [torch.randint(0, 1 << 30, (8001 * 6003,), dtype=torch.int32,
                          device="cuda") for _ in streams]
    want = [b.view(8001, 6003).t().reshape(-1) for b in bufs]
    torch.cuda.synchronize()
    for s, b in zip(streams, bufs):
        lm.transpose_100(b, 8001, 6003, 1, stream=s)
        lm.transpose_100(b, 6003, 8001, 1, stream=s)
        lm.transpose_100(b, 8001, 6003, 1, stream=s)
    torch.cuda.synchronize()
    for b, w in zip(bufs, want):
        assert torch.equal(b, w)
    assert lm.lib().lm_device_status(None) == 0


@pytest.mark.parametrize("T,a,B,e", [(3, 6001, 6003, 4), (2, 15159, 10641, 1),
                                     (17, 4001, 4201, 8), (2, 9001, 9003, 2)])
def test_instances(T, a, B, e):
    """Large instances one after another, each at its own place in 16 bytes."""
    n = a * B * e
    raw = torch.randint(0, 256, (T * n,), dtype=torch.uint8, device="cuda")
    want = raw.view(T, a, B, e).transpose(1, 2).reshape(-1)
    lm.prof_collect()
    lm.prof_enable(True)
    lm.transpose_0100(raw, T, a, B, 1, elem_bytes=e)
    torch.cuda.synchronize()
    lm.prof_enable(False)
    assert set(lm.prof_collect()) == {"wave", "suffix_copy"}
    assert torch.equal(raw, want)


@pytest.mark.parametrize("a,B,e", [(9000001, 5, 4), (40001, 701, 4),
                                   (24001, 5001, 1), (3000001, 33, 2)])
def test_staged_is_left(a, B, e):
    """Below the sizes of the ordered form, and rows too short for it."""
    _check(a, B, 1, e, wave=False)


@pytest.mark.parametrize("a,B,ran", [
    (28775, 4005, {"stash_save", "stash_wave"}),
    (28776, 4005, {"wave", "suffix_copy"}),  # whole vectors
    (28775, 4001, {"wave", "suffix_copy"}),  # rows 2 bytes past some
    (22999, 5005, {"wave", "suffix_copy"}),
    (40001, 3005, {"wave", "suffix_copy"}),  # more rows than the stash takes
])
def test_tall_half_words(a, B, ran):
    """Which of the two forms at 3 x payload takes tall matrices."""
    x = torch.randint(-30000, 30000, (a, B), dtype=torch.int16, device="cuda")
    want = x.t().reshape(-1)
    lm.transpose_100(x.clone(), a, B, 1)  # (plans are kept per shape)
    lm.prof_collect()
    lm.prof_enable(True)
    lm.transpose_100(x, a, B, 1)
    torch.cuda.synchronize()
    lm.prof_enable(False)
    assert set(lm.prof_collect()) == ran
    assert torch.equal(x.view(-1), want)


# forward and backward, blocks of whole vectors and ragged ones
@pytest.mark.parametrize("a,B,b,e", [(8192, 8191, 1, 4), (8191, 4097, 1, 4),
                                     (125000, 101, 8, 4), (40001, 3001, 1, 1),
                                     (300001, 301, 1, 2)])
def test_wait_that_runs_out_is_reported(a, B, b, e):
    """Blocks that wait for one block more of an earlier step than there are
    give up after 20 ms, as whole warps; the call reports it, and the next ones
    work."""
    x = torch.randint(0, 256, (a * B * b * e,), dtype=torch.uint8, device="cuda")
    want = x.view(a, B, b * e).transpose(0, 1).reshape(-1)
    for _ in range(2):
        y = x.clone()
        assert lm.lib().lm_debug_wave_stall(None, y.data_ptr(), e, a, B, b,
                                            20_000_000) is True
        assert "timed out" in lm.last_error()
    assert lm.lib().lm_device_status(None) == 0
    lm.transpose_100(x, a, B, b, elem_bytes=e)
    torch.cuda.synchronize()
    assert torch.equal(x, want)
    assert lm.lib().lm_device_status(None) == 0
