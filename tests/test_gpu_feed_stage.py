"""Feeds of a predictor between two forwards: one input fed again and again, more inputs and bytes than the staging buffer
takes at once, small and long arrays in turn, feeds from host and device memory in turn, reshapes, and a fed blob read back.
The last data fed are the ones the net sees."""
import numpy as np
import pytest
import torch

import pkg

pytestmark = pytest.mark.gpu


def _predictor(n_inputs):
    pkg.load()
    from x_deeplearning_b200 import blaze_api as api
    ops = [api.constant_text("one", np.ones((1, 1)), 1)]
    ops += [api.op_text("Add", ["x%d" % i, "one"], ["y%d" % i]) for i in range(n_inputs)]
    mgr = api.PredictorManager()
    mgr.load_model_text(api.netdef_text(ops, [("x%d" % i, 1) for i in range(n_inputs)], [("y%d" % i, 1) for i in range(n_inputs)]))
    return mgr, mgr.create_predictor(device_type=1, device_id=0)


def _value(i, shape):
    return (np.arange(np.prod(shape)).reshape(shape) % 251 + i).astype(np.float32)


@pytest.mark.parametrize("cols", [1, 250, 8192])
def test_one_input_fed_again_and_again(cols):
    mgr, p = _predictor(1)
    p.reshape("x0", (1, cols))
    for _ in range(2):
        for i in range(40 if cols > 1000 else 2500):                 # 8192 floats: the longest array that is staged
            a = _value(i, (1, cols))
            p.feed_raw("x0", a.ctypes.data, a.nbytes)
        p.forward()
        assert np.array_equal(p.output("y0"), a + 1)
    p.close(); mgr.close()


@pytest.mark.parametrize("n,cols", [(140, 50), (40, 8192)])
def test_more_inputs_and_bytes_than_the_stage_takes_at_once(n, cols):
    mgr, p = _predictor(n)
    for k in range(3):
        data = [_value(i + k, (1, cols)) for i in range(n)]
        for i, a in enumerate(data):
            p.feed("x%d" % i, a)
        p.forward()
        for i, a in enumerate(data):
            assert np.array_equal(p.output("y%d" % i), a + 1)
    p.close(); mgr.close()


def test_host_and_device_feeds_in_turn():
    mgr, p = _predictor(1)
    host, dev = _value(1, (4, 300)), torch.from_numpy(_value(5, (4, 300))).cuda()
    torch.cuda.synchronize()
    p.reshape("x0", host.shape)
    for last in ("device", "host"):
        for i in range(600):
            p.feed_raw("x0", host.ctypes.data, host.nbytes)
            if last == "device" or i < 599:
                p.feed_device("x0", dev.data_ptr(), host.nbytes)
        p.forward()
        assert np.array_equal(p.output("y0"), (dev.cpu().numpy() if last == "device" else host) + 1)
    p.close(); mgr.close()


def test_small_and_long_arrays_and_reshapes_between_feeds():
    mgr, p = _predictor(2)
    shapes = [(2, 100), (300, 100), (1, 7), (5, 1000), (90, 91), (3, 3)]      # some staged, some beyond the staged length
    other = _value(9, (3, 50))
    p.feed("x1", other)
    for i, sh in enumerate(shapes):
        a = _value(i, sh)
        p.feed("x0", a)
        assert np.array_equal(p.output("x0"), a)                              # a fed blob reads back before any forward
    p.forward()
    assert np.array_equal(p.output("y0"), a + 1) and np.array_equal(p.output("y1"), other + 1)
    b = _value(77, shapes[-1])
    p.feed("x0", b)                                                           # the other input keeps what it holds
    p.forward()
    assert np.array_equal(p.output("y0"), b + 1) and np.array_equal(p.output("y1"), other + 1)
    ptr, n = p.output_device("x0")
    assert n == b.nbytes and ptr
    p.close(); mgr.close()
