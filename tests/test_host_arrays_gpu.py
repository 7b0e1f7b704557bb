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


@pytest.mark.parametrize("asked_for", ["value_info", "synchronize"])
@pytest.mark.parametrize("rows", [1, 200])
def test_fed_input_is_on_the_device_before_the_run(cuda, asked_for, rows):
    """The address of an input that has just been fed: its data is there behind synchronize, and behind the stream's work once the address is out."""
    import torch
    cols = 1024
    inst = _doubler(cols)
    r = np.random.default_rng(rows)
    inst.run({"x": r.standard_normal((rows, cols), dtype=np.float32)})
    x = r.standard_normal((rows, cols), dtype=np.float32)
    ptr = inst.value_info("x")[2]
    inst.set_input("x", x)
    if asked_for == "value_info":
        ptr = inst.value_info("x")[2]
        torch.cuda.synchronize()
    else:
        inst.synchronize()

    class Array:
        __cuda_array_interface__ = {"version": 3, "data": (ptr, False), "shape": x.shape, "typestr": "<f4", "strides": None}

    assert np.array_equal(torch.as_tensor(Array(), device="cuda").cpu().numpy(), x)


def test_threads_read_one_instance(cuda):
    """Two threads read outputs of different shapes, types and sizes of one instance at the same time."""
    from concurrent.futures import ThreadPoolExecutor
    from rmlk_b200.runtime import ModelInstance
    g = GraphSpec()
    g.input("x", np.float32, [0, 1024])
    g.input("n", np.int64, [0])
    g.op("Add", ["x", "x"], "y")
    g.op("Add", ["n", "n"], "m")
    g.output("y")
    g.output("m")
    inst = ModelInstance(g.to_runtime())
    x, n = np.random.default_rng(1).standard_normal((150, 1024), dtype=np.float32), np.arange(3000, dtype=np.int64)
    inst.run({"x": x, "n": n})

    def reads(name, want):
        return all((lambda got: got.dtype == want.dtype and np.array_equal(got, want))(inst.read(name)) for _ in range(300))

    with ThreadPoolExecutor(4) as pool:
        jobs = [pool.submit(reads, *a) for a in (("y", 2 * x), ("m", 2 * n), ("y", 2 * x), ("m", 2 * n))]
        assert all(j.result() for j in jobs)


def test_reading_a_shape_reports_the_errors_of_the_run(cuda):
    from rmlk_b200.runtime import InferenceError, ModelInstance
    g = GraphSpec()
    g.input("data", np.float32, [0, 4])
    g.input("at", np.int64, [0])
    g.op("Gather", ["data", "at"], "y", axis=0)
    g.op("Shape", ["y"], "shape")
    g.op("Reshape", ["y", "shape"], "z")
    g.output("z")
    inst = ModelInstance(g.to_runtime())
    at = np.zeros(100, np.int64)
    for name, value in (("data", np.zeros((8, 4), np.float32)), ("at", at)):
        inst.set_input(name, value)
    inst.launch()
    assert inst.read("shape").tolist() == [100, 4]
    at[70] = 9  # out of range: seen by the kernel, which writes nothing there
    for name, value in (("data", np.zeros((8, 4), np.float32)), ("at", at)):
        inst.set_input(name, value)
    inst.launch()
    with pytest.raises(InferenceError):
        inst.read("shape")
