"""Every size of the Fr transform, with counts that leave a block's last
transforms unused, in place as well."""
import numpy as np
import pytest

import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log_m", range(1, 10))
@pytest.mark.parametrize("inverse", [0, 1])
def test_fr_fft_every_size(engine, log_m, inverse):
    m = 1 << log_m
    count = 1024 // m + 3
    x = O.seeded_fr(40 + log_m, count * m).reshape(count, m, 4)
    x[0, :] = O.int_to_limbs(O.R - 1, 4)
    d = engine.to_device(x)
    out = engine.empty(x.shape)
    exp = O.fr_fft(x, inverse=bool(inverse))
    engine.call("fr_fft_n", engine._ptr(out), engine._ptr(d), log_m, count, inverse, engine._stream())
    assert np.array_equal(engine.to_host(out), exp)
    engine.call("fr_fft_n", engine._ptr(d), engine._ptr(d), log_m, count, inverse, engine._stream())
    assert np.array_equal(engine.to_host(d), exp)


@pytest.mark.parametrize("log_m", range(3, 10))
@pytest.mark.parametrize("past", [0, 1])
def test_fr_fft_around_the_line(engine, log_m, past):
    """The largest count of the kernel for few transforms, and one more."""
    m = 1 << log_m
    count = min(148 * 12, 148 * 1024 // m) + past
    x = O.seeded_fr(60 + log_m, count * m).reshape(count, m, 4)
    d = engine.to_device(x)
    for inverse in (0, 1):
        out = engine.empty(x.shape)
        engine.call("fr_fft_n", engine._ptr(out), engine._ptr(d), log_m, count, inverse, engine._stream())
        assert np.array_equal(engine.to_host(out), O.fr_fft(x, inverse=bool(inverse)))


# values an SM that each size leaves to the kernel for few transforms, forward and inverse
LINES = [[8, 80, 176, 400, 672, 944, 1472, 1536, 1024], [8, 64, 176, 400, 816, 1312, 1648, 1600, 1536]]


@pytest.mark.parametrize("log_m", range(1, 10))
@pytest.mark.parametrize("inverse", [0, 1])
def test_fr_fft_on_both_sides_of_its_line(engine, log_m, inverse):
    import torch
    m = 1 << log_m
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for count in (sms * LINES[inverse][log_m - 1] // m + k for k in (0, 1)):
        x = O.seeded_fr(80 + log_m, count * m).reshape(count, m, 4)
        d = engine.to_device(x)
        exp = O.fr_fft(x, inverse=bool(inverse))
        engine.call("fr_fft_n", engine._ptr(d), engine._ptr(d), log_m, count, inverse, engine._stream())
        assert np.array_equal(engine.to_host(d), exp)
