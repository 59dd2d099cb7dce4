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
    assert lib.fk20_default_set(63, engine.FK20_OPT_FUSED_FFT, 1) == engine.FK20_ENODEV


@pytest.mark.parametrize("inverse", [0, 1])
@pytest.mark.parametrize("log_m,count", [(1, 1), (1, 33), (1, 5000), (2, 1), (2, 40), (2, 5000), (3, 4097), (3, 65536 + 40),
                                         (4, 2050)])
def test_short_transforms_by_stages_and_in_passes(engine, log_m, count, inverse):
    """Two points, and four forward, go by radix-2 stages; longer ones by plans, 2^19
    points of rows a pass.  Blocks of distinct transforms repeat, so that only the
    first needs the oracle."""
    import torch
    m, distinct = 1 << log_m, min(count, 24)
    x = points(40 + log_m, distinct * m).reshape(distinct, m, 18)
    src = engine.to_device(x).repeat((count + distinct - 1) // distinct, 1, 1)[:count].contiguous()
    out = engine.empty((count, m, 18))
    engine.call("g1p_fft_n", engine._ptr(out), engine._ptr(src), log_m, count, inverse, engine._stream())
    torch.cuda.synchronize()
    whole = count // distinct * distinct
    blocks = out[:whole].reshape(-1, distinct, m, 18)
    assert (blocks == blocks[0]).all() and (out[whole:] == blocks[0][:count - whole]).all()
    assert np.array_equal(normalized(engine, out[:distinct]), O.g1_fft(x, inverse=bool(inverse)))
    engine.call("g1p_fft_n", engine._ptr(src), engine._ptr(src), log_m, count, inverse, engine._stream())
    assert torch.equal(src, out)  # in place


@pytest.mark.parametrize("log_m,inverse", [(1, 0), (1, 1), (2, 0), (2, 1), (3, 0)])
def test_no_allocation_entry_gives_the_same_words(engine, log_m, inverse):
    """Also where the points of both are not normalised."""
    import torch
    m = 1 << log_m
    src = engine.to_device(points(50 + log_m, 37 * m).reshape(37, m, 18))
    a, b = engine.empty(src.shape), engine.empty(src.shape)
    for call, out in (("g1p_fft_n", a), ("g1p_fft_noalloc", b)):
        engine.call(call, engine._ptr(out), engine._ptr(src), log_m, 37, inverse, engine._stream())
    torch.cuda.synchronize()
    assert torch.equal(a, b)
    raw = log_m == 1 or (log_m == 2 and not inverse)
    assert raw == bool((a.reshape(-1, 18)[:, 12] != 1).any())


def test_transforms_without_room_for_their_arena(engine):
    """The device allocations of the arena fail (injected): the transforms go by
    stages and give the same words; only when those fail too do they refuse."""
    import torch
    dev, lib = torch.cuda.current_device(), engine.lib()
    x = points(61, 40 * 512).reshape(40, 512, 18)
    src = engine.to_device(x)
    calls = [("g1p_fft", 512, 40, ()), ("g1p_ift", 512, 40, ()), ("fk20_hext_fft2h_fft", 512, 33, ()),
             ("g1p_fft_n", 8, 700, (3, 0)), ("g1p_fft_n", 4, 700, (2, 1))]

    def run(name, m, count, first):
        out = engine.empty((count, m, 18))
        args = first and (first[0], count, first[1]) or (count,)
        engine.call(name, engine._ptr(out), engine._ptr(src), *args, engine._stream())
        torch.cuda.synchronize()
        return out

    try:
        for c in calls:
            good = run(*c)
            assert lib.fk20_default_release(dev) == 0
            assert lib.fk20_test_fail_allocations(1) == 0
            assert torch.equal(run(*c), good), c
            assert lib.fk20_default_release(dev) == 0
            assert lib.fk20_test_fail_allocations(2) == 0
            with pytest.raises(engine.Fk20Error) as err:
                run(*c)
            assert err.value.code == engine.FK20_ENOMEM
            assert torch.equal(run(*c), good), c
    finally:
        lib.fk20_test_fail_allocations(0)


@pytest.mark.parametrize("log_m,inverse", [(3, 0), (6, 1), (9, 0)])
def test_transforms_level_by_level_give_the_same_words(engine, log_m, inverse):
    """FK20_OPT_FUSED_FFT 0 on the default context: a launch per level, 300 rows in
    chunks of groups."""
    import torch
    dev, lib, m = torch.cuda.current_device(), engine.lib(), 1 << log_m
    src = engine.to_device(points(70 + log_m, 6 * m).reshape(6, m, 18)).repeat(50, 1, 1)
    a, b = engine.empty(src.shape), engine.empty(src.shape)
    try:
        for fused, out in ((1, a), (0, b)):
            assert lib.fk20_default_set(dev, engine.FK20_OPT_FUSED_FFT, fused) == 0
            engine.call("g1p_fft_n", engine._ptr(out), engine._ptr(src), log_m, 300, inverse, engine._stream())
    finally:
        lib.fk20_default_set(dev, engine.FK20_OPT_FUSED_FFT, 1)
    assert lib.fk20_default_status(dev) == 0
    assert torch.equal(a, b)
