"""A carried cache's buffer is taken over by the next sequence when it is large enough."""
import numpy as np
import pytest

from rmlk_b200.graphspec import GraphSpec

pytestmark = pytest.mark.gpu


def _instance(kv, d):
    from rmlk_b200.runtime import ModelInstance
    g = GraphSpec()
    g.input("new", np.float32, [0, kv, 0, d])
    g.input("past", np.float32, [0, kv, 0, d])
    g.op("Concat", ["past", "new"], "present", axis=2)
    g.output("present")
    inst = ModelInstance(g.to_runtime())
    inst.bind("present", "past")
    return inst


# (batch, rows fed, steps of one row): the second and later sequences are smaller, equal, larger, differently shaped and empty
@pytest.mark.parametrize("sequences", [
    [(2, 40, 3), (2, 40, 3), (2, 7, 2), (1, 100, 2), (5, 30, 4), (2, 0, 3)],
    [(1, 0, 1), (1, 63, 3), (1, 64, 70), (1, 200, 1), (3, 1, 1)],
])
def test_sequences_share_one_buffer(cuda, sequences):
    from rmlk_b200 import dtypes as dt
    import torch
    kv, d = 3, 8
    inst = _instance(kv, d)
    r = np.random.default_rng(5)
    for i, (b, t, steps) in enumerate(sequences):
        cache = r.standard_normal((b, kv, t, d), dtype=np.float32)
        on_device = torch.from_numpy(cache).to(cuda)
        if i % 2 and t:
            inst.set_input_ptr("past", dt.F32, [b, kv, t, d], on_device.data_ptr(), True)
        else:
            inst.set_input("past", cache)
        for _ in range(steps):
            new = r.standard_normal((b, kv, 1, d), dtype=np.float32)
            inst.set_input("new", new)
            inst.launch()
            cache = np.concatenate([cache, new], axis=2)
        assert np.array_equal(inst.read("present"), cache), (i, b, t)


def test_a_cache_fed_from_inside_its_own_buffer(cuda):
    """One head: the carried view is dense and its address is handed out; rows fed from the middle of it are moved intact."""
    from rmlk_b200 import dtypes as dt
    d = 8
    inst = _instance(1, d)
    r = np.random.default_rng(6)
    cache = r.standard_normal((1, 1, 50, d), dtype=np.float32)
    inst.set_input("past", cache)
    new = r.standard_normal((1, 1, 2, d), dtype=np.float32)
    inst.set_input("new", new)
    inst.launch()
    cache = np.concatenate([cache, new], axis=2)
    _, shape, ptr = inst.value_info("present")
    assert shape == [1, 1, 52, d] and ptr
    inst.set_input_ptr("past", dt.F32, [1, 1, 40, d], ptr + 12 * d * 4, True)
    inst.set_input("new", new)
    inst.launch()
    assert np.array_equal(inst.read("present"), np.concatenate([cache[:, :, 12:], new], axis=2))
