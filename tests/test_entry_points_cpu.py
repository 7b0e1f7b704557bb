"""Entry points of the runtime, as far as a host without a GPU can look at them."""
import os
import re

import rmlk_b200

CSRC = os.path.join(os.path.dirname(rmlk_b200.__file__), "csrc", "runtime", "runtime.cpp")


def test_entry_points_that_launch_set_the_device():
    """A kernel launch on a stream of another device fails; copies there do not, so an entry point that comes to launch one needs its device made
    current.  (Two devices in one process: what is looked at here is the source.)"""
    with open(CSRC) as f:
        source = f.read()
    bodies = {}
    for part in source.split('extern "C" ')[1:]:
        name = re.match(r"[\w \*]*?(rmlk_instance_\w+)\(", part)
        if name:
            bodies[name.group(1)] = part
    assert {"rmlk_instance_read", "rmlk_instance_value_info", "rmlk_instance_set_input", "rmlk_instance_run"} <= set(bodies)
    launching = re.compile(r"strided_copy|settle_host_only|flush_uploads|read_to_host|feed_host|host_download|host_upload")
    checked = 0
    for name, body in bodies.items():
        at = launching.search(body)
        if at:
            checked += 1
            assert "cudaSetDevice" in body[: at.start()], name
    assert checked >= 3
    run = re.search(r"void Instance::run\(\) \{(.*?)\n\}", source, re.S).group(1)
    assert run.index("cudaSetDevice") < run.index("flush_uploads")


def test_dims_of_any_integer_type():
    import numpy as np
    import torch
    from rmlk_b200 import kernels, runtime
    for make in (runtime._i64, kernels._i64):
        for dims in ([], [3], (2, 5), list(range(12)), np.arange(4), [np.int32(7), 2], torch.Size([4, 6]), [torch.tensor(9), 1], [True, 2.0]):
            assert list(make(dims))[: len(dims)] == [int(v) for v in dims]


def test_every_handle_is_passed_whole():
    """ctypes cuts an int argument of a function without argtypes to 32 bits: a handle that lies higher would arrive broken."""
    import inspect
    from rmlk_b200 import runtime
    library = runtime._rt()
    names = set(re.findall(r"\.(rmlk_(?:graph|instance)_\w+)\(", inspect.getsource(runtime)))
    assert "rmlk_instance_stream_output" in names
    for name in names - {"rmlk_graph_create"}:
        assert getattr(library, name).argtypes, name
