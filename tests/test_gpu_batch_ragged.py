"""Batches whose staged items mix blocks of 1- and 2-byte elements that start
anywhere in a 16-byte vector (k_batch_gather<2, 1, 0>) with other items, and
large jobs staged beside them."""
import pytest

torch = pytest.importorskip("torch")

from libmarshal_gb300 import lm

pytestmark = pytest.mark.gpu

DT = {1: torch.uint8, 2: torch.int16, 4: torch.int32, 8: torch.int64}


def _run(shapes, offset=0):
    """shapes: (rows, columns, element bytes) of transpositions."""
    jobs, keep = [], []
    for k, (h, w, e) in enumerate(shapes):
        g = torch.Generator(device="cuda").manual_seed(k + h + offset)
        raw = torch.randint(0, 256, (h * w * e + 32,), dtype=torch.uint8,
                            device="cuda", generator=g)
        off = offset * e % 16
        src = raw[off:off + h * w * e].clone().view(DT[e]).view(h, w)
        want = raw.clone()
        want[off:off + h * w * e] = src.t().contiguous().view(-1).view(torch.uint8)
        jobs.append(lm.job(raw.data_ptr() + off, lm.OP_TRANSPOSE, (h, w),
                           elem_bytes=e))
        keep.append((raw, want))
    b = lm.Batch()
    b.run(jobs)
    torch.cuda.synchronize()
    for (raw, want), shape in zip(keep, shapes):
        assert torch.equal(raw, want), shape
    return b.stats()


@pytest.mark.parametrize("offset", [0, 1])
def test_mixed(offset):
    shapes = [(1101, 701, 1), (2049, 517, 1), (4095, 63, 1), (1500, 1500, 2),
              (3001, 999, 2), (4093, 120, 2), (1300, 333, 4), (2000, 401, 8),
              (1026, 2051, 1), (1025, 1030, 2)]
    st = _run(shapes, offset)
    assert st["staged_jobs"] >= 8


def test_large_beside():
    st = _run([(2143, 2145, 4), (1201, 2245, 8), (1101, 701, 1), (33, 65, 2)])
    assert st["large_jobs"] == 2
