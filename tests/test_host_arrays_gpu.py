"""Host arrays on their way in and out: what the caller does with them afterwards, and what was enqueued before them."""
import numpy as np
import pytest

from rmlk_b200.graphspec import GraphSpec

pytestmark = pytest.mark.gpu


def _doubler(cols, stream=None):
    from rmlk_b200.runtime import ModelInstance
    g = GraphSpec()
    g.input("x", np.float32, [0, cols])
    g.op("Add", ["x", "x"], "y")
    g.output("y")
    return ModelInstance(g.to_runtime(), stream=stream)


# below and above the sizes at which transfers take another way
@pytest.mark.parametrize("rows", [1, 64, 700, 2000])
def test_results_may_be_changed_after_they_were_fed(cuda, rows):
    import torch
    cols = 1024
    busy = torch.cuda.Stream()
    first, second = _doubler(cols), _doubler(cols, busy.cuda_stream)
    x = np.random.default_rng(rows).standard_normal((rows, cols), dtype=np.float32)
    y = first.run({"x": x})["y"]
    assert not torch.from_numpy(y).is_pinned()
    with torch.cuda.stream(busy):
        torch.cuda._sleep(20_000_000)  # about 10 ms: whatever is fed now is still to come
    second.set_input("x", y)
    second.launch()
    y += 1
    del y
    first.run({"x": x + 5})  # (takes the memory that was given back)
    assert np.array_equal(second.read("y"), 4 * x)


@pytest.mark.parametrize("rows", [1, 8, 9, 200, 300])
def test_pinned_input_is_read_in_stream_order(cuda, rows):
    """What the stream writes into pinned memory before a run is what the run is fed, at every size."""
    import torch
    from rmlk_b200 import dtypes as dt
    cols = 1024
    stream = torch.cuda.Stream()
    inst = _doubler(cols, stream.cuda_stream)
    pinned = torch.zeros(rows, cols, pin_memory=True)
    x = torch.randn(rows, cols, device=cuda)
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(20_000_000)
        pinned.copy_(x, non_blocking=True)
    inst.set_input_ptr("x", dt.F32, [rows, cols], pinned.data_ptr(), False)
    inst.launch()
    assert np.array_equal(inst.read("y"), 2 * x.cpu().numpy())
