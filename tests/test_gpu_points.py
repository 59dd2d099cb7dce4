"""Transforms of points (g1p_fft and its relatives, fk20_hext_fft2h_fft) on the
default context, beyond the sizes of test_gpu_fft.py."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


def points(seed, count):
    return O.g1_op("mul", np.repeat(O.g1_generator().reshape(1, 18), count, 0), O.seeded_fr(seed, count))


def normalized(engine, t):
    a = engine.to_host(t)
    return O.g1_normalize(a.reshape(-1, 18)).reshape(a.shape)


@pytest.mark.parametrize("call", ["g1p_fft_n", "fk20_hext_fft2h_fft"])
def test_abandoned_transform_is_reported_and_refuses_nothing(engine, call):
    """A bounded wait of a transform runs out (one task publishes nothing, as a
    host-set hook says): the status call reports it once, also after a later
    call that succeeded, and that call is not refused."""
    import torch
    dev = torch.cuda.current_device()
    lib = engine.lib()
    x = points(31, 40 * 32).reshape(40, 32, 18)
    src, out = engine.to_device(x), engine.empty(x.shape)
    y = engine.to_device(points(32, 3 * 512).reshape(3, 512, 18))
    h = engine.empty((3, 512, 18))

    def transform():
        engine.call("g1p_fft_n", engine._ptr(out), engine._ptr(src), 5, 40, 0, engine._stream())

    transform()
    assert lib.fk20_default_status(dev) == 0
    assert lib.fk20_default_set(dev, engine.FK20_OPT_WAIT_LIMIT, 1 << 12) == 0
    assert lib.fk20_default_set(dev, engine.FK20_OPT_TEST_UNPUBLISHED_TASK, 3) == 0
    try:
        if call == "g1p_fft_n":
            transform()
        else:
            engine.call(call, engine._ptr(h), engine._ptr(y), 3, engine._stream())
    finally:
        assert lib.fk20_default_set(dev, engine.FK20_OPT_TEST_UNPUBLISHED_TASK, -1) == 0
        assert lib.fk20_default_set(dev, engine.FK20_OPT_WAIT_LIMIT, 0) == 0
    transform()
    torch.cuda.synchronize()
    assert np.array_equal(normalized(engine, out), O.g1_fft(x))
    assert lib.fk20_default_status(dev) == engine.FK20_ETIMEOUT
    assert lib.fk20_default_status(dev) == 0
    assert lib.fk20_default_status(-1) == engine.FK20_EINVAL
    assert lib.fk20_default_set(dev, 99, 0) == engine.FK20_EINVAL
