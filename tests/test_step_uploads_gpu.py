"""What a step copies to the device before its kernels: changed block-table entries, in one copy or in several, and the events behind them."""
import numpy as np
import pytest
import torch

from rocmforge_b200.cache import KVRequest
from rocmforge_b200.cache.sequence_cache import KVGroup, upload_spans
from rocmforge_b200.kernels import _ffi

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("slots,width", [(6, 8), (5, 6000)])          # changes near each other, and rows too far apart for one copy
def test_device_table_after_uploads(slots, width):
    group = KVGroup(KVRequest(1, 16), [0], 400, slots, width, torch.float32, torch.device(DEV))
    want = np.zeros((slots, width), dtype=np.int64)
    rng = np.random.default_rng(width)
    several = set()
    for step in range(30):                                # each upload reuses the staging buffer and the event of the one before
        for slot in rng.choice(slots, size=2, replace=False):
            if rng.random() < 0.3:
                group.release(int(slot))
            else:
                start = int(rng.integers(0, min(width, 64))) * 64
                group.ensure(int(slot), start, min(width * 64, start + int(rng.integers(1, 200))))
        dirty = {s: list(r) for s, r in group._dirty.items()}
        if dirty:
            spans = upload_spans(dirty, width)
            several.add(len(spans) > 1)
            for a, b in spans:
                want.reshape(-1)[a:b] = group.table.reshape(-1)[a:b]
        group.upload()
        assert not group._dirty
        assert np.array_equal(group.table_dev.cpu().numpy(), want)
        held = group.table >= 0
        assert np.array_equal(want[held], group.table[held])          # every page that a sequence holds is named on the device
        assert (want[~held] <= 0).all()                               # ... and no other one but page 0, which nothing has written over
    assert (True in several) == (width == 6000)


def test_events_are_recorded_on_the_current_stream():
    """``record`` keeps a Stream object by the stream's handle: each stream and each event must come out as with ``event.record()``."""
    x = torch.zeros((64 << 20,), device=DEV)
    streams = [torch.cuda.current_stream(), torch.cuda.Stream(), torch.cuda.Stream()]
    for turn in range(3):
        for s in streams:
            with torch.cuda.stream(s):
                start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                _ffi.record(start)
                for _ in range(4):
                    x.add_(1.0)                           # some hundred microseconds of work on this stream
                _ffi.record(end)
            end.synchronize()
            assert end.query() and start.elapsed_time(end) > 0.05
            torch.cuda.synchronize()
    keep = dict(_ffi._streams)
    assert all(s.cuda_stream == handle for (_, handle), s in keep.items())
    for i in range(200):                                  # more streams than are kept: the notes stay bounded
        with torch.cuda.stream(torch.cuda.Stream(priority=-(i % 2))):
            _ffi.record(torch.cuda.Event())
    torch.cuda.synchronize()
    assert len(_ffi._streams) <= 64
