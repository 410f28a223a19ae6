"""Calls from several host threads at once, each on its own stream and buffers,
whose kernels are the same but for their sizes and share what the library keeps
for the process."""
import threading

import pytest

torch = pytest.importorskip("torch")

from libmarshal_gb300 import lm

pytestmark = pytest.mark.gpu


def _threads(n, work):
    """work(k, stream) in n threads that start together."""
    errors = []
    gate = threading.Barrier(n)

    def body(k):
        try:
            s = torch.cuda.Stream()
            with torch.cuda.stream(s):
                gate.wait()
                work(k, s)
        except Exception as ex:  # noqa: BLE001
            errors.append((k, repr(ex)))

    ts = [threading.Thread(target=body, args=(k,)) for k in range(n)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    torch.cuda.synchronize()
    assert not errors, errors[:3]


@pytest.mark.parametrize("e", [4, 8])
def test_squares(e):
    """Squares whose blocks take shared memory of different sizes."""
    sizes = (333, 700, 8192, 1000, 5000, 400)
    dt = {4: torch.int32, 8: torch.int64}[e]
    xs = [torch.randint(0, 1 << 30, (n, n), dtype=dt, device="cuda")
          for n in sizes]
    want = [x.t().contiguous() for x in xs]
    torch.cuda.synchronize()

    def work(k, s):
        for i in range(5):
            lm.transpose_100(xs[k], sizes[k], sizes[k], 1, stream=s)

    _threads(len(sizes), work)
    for x, w in zip(xs, want):
        assert torch.equal(x, w)
    assert lm.lib().lm_device_status(None) == 0


@pytest.mark.parametrize("method", [0, 3, 6])  # planner, stash, staged
def test_forms_of_large_matrices(method):
    """One form's kernels with blocks and steps of different sizes."""
    shapes = [(8001, 4003, 4), (12000, 1601, 4), (9001, 6007, 2),
              (9600, 801, 8), (16001, 3001, 1), (10240, 640, 4)]
    dt = {1: torch.uint8, 2: torch.int16, 4: torch.int32, 8: torch.int64}
    xs = [torch.randint(0, 100, (a, b), device="cuda").to(dt[e])
          for a, b, e in shapes]
    want = [x.t().reshape(-1) for x in xs]
    torch.cuda.synchronize()

    def work(k, s):
        a, b, e = shapes[k]
        for i in range(3):
            d = xs[k].clone()
            lm.transpose_0100(d, 1, a, b, 1, method=method, stream=s)
            assert torch.equal(d.view(-1), want[k])

    _threads(len(shapes), work)
    assert lm.lib().lm_device_status(None) == 0


def test_padding_flags_of_many_threads():
    """Twenty threads, more than blocks of flags are kept, pad and unpad their
    own buffers with task counts that go up and down, on their own streams."""
    shapes = [(1000, 600, 1010), (7, 9, 8), (300, 40000, 301), (50, 3001, 64),
              (4000, 101, 4096)]

    def work(k, s):
        for i in range(6):
            x, y, pad = shapes[(k + i) % len(shapes)]
            src = torch.arange(k, k + y * x, dtype=torch.int32, device="cuda")
            d = torch.full((y * pad,), -1, dtype=torch.int32, device="cuda")
            d[:y * x] = src
            lm.padding(d, x, y, pad, stream=s)
            want = torch.zeros((y, pad), dtype=torch.int32, device="cuda")
            want[:, :x] = src.view(y, x)
            assert torch.equal(d.view(y, pad), want)
            lm.unpadding(d, x, y, pad, stream=s)
            assert torch.equal(d[:y * x], src)
            assert not d[y * x:].any()

    _threads(20, work)


def test_padding_about_the_kept_flags():
    """Calls with a task less and more than a kept block has words for, and
    small ones between them; and the call after one that timed out, whose block
    is not used again."""
    task = 16 * 1024
    small = torch.zeros(1010 * 600, dtype=torch.int32, device="cuda")
    for tasks in (16 * 1024 - 2, 16 * 1024 - 1, 16 * 1024 - 2, 20000):
        pad = 4096  # one row of floats is one task
        x = pad - 3
        d = torch.zeros(tasks * pad, dtype=torch.int32, device="cuda")
        src = torch.randint(1, 1 << 30, (tasks * x,), dtype=torch.int32,
                            device="cuda")
        assert d.numel() * 4 == tasks * task
        d[:tasks * x] = src
        lm.padding(d, x, tasks, pad)
        assert torch.equal(d.view(tasks, pad)[:, :x], src.view(tasks, x))
        assert not d.view(tasks, pad)[:, x:].any()
        small.fill_(7)
        lm.padding(small, 1000, 600, 1010)
        assert int(small.sum()) == 7 * 1000 * 600
        assert lm.lib().lm_debug_pad_stall(None, small.data_ptr(), 4, 1000, 600,
                                           1010, 0, 3, 20_000_000) is True
        assert "timed out" in lm.last_error()
        lm.unpadding(d, x, tasks, pad)
        assert torch.equal(d[:tasks * x], src)
        assert not d[tasks * x:].any()
        del d, src
