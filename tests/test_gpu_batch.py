"""Batched uneven channels: one graph launch per step advances every
channel exactly as the channel would alone; the autotuner keeps the state."""
import math

import numpy as np
import pytest

from tests.conftest import relerr

pytestmark = pytest.mark.gpu

CFGS = [dict(nx=32, ny=32, nz=48, ren=2500.0), dict(nx=112, ny=48, nz=64, ren=4000.0),
        dict(nx=64, ny=16, nz=176, ren=3000.0), dict(nx=48, ny=64, nz=32, ren=5500.0)]


def _need_gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def test_batch_step_equals_single_channels():
    _need_gpu()
    from chapsim1ww_b200 import ChannelBatch, TGChannel
    b = ChannelBatch(CFGS)
    b.init_random(seed=3, amp=0.1, project=True)
    b.step(3)
    b.sync()
    assert b.kernels_per_step() == 3 * 10 * len(CFGS)  # 10 kernels per FP64 substep
    for i, c in enumerate(CFGS):
        s = TGChannel(**c)
        s.random_fl_fld_tg(3 + i, 0.1, project=True)
        s.step(3)
        for n in ("u", "v", "w", "p"):
            assert np.array_equal(s.get_field(n), b.channels[i].get_field(n)), (i, n)
        assert b.channels[i].divgck_tg() < 1e-11


def test_autotune_keeps_state_and_results():
    _need_gpu()
    from chapsim1ww_b200 import ChannelBatch
    b = ChannelBatch(CFGS[:2])
    b.init_random(seed=5, amp=0.1, project=True)
    before = [b.channels[i].get_field("u") for i in range(2)]
    b.autotune(reps=3)
    for i in range(2):
        assert np.array_equal(before[i], b.channels[i].get_field("u"))
    ref = ChannelBatch(CFGS[:2])
    ref.init_random(seed=5, amp=0.1, project=True)
    b.step(2)
    ref.step(2)
    b.sync()
    ref.sync()
    for i in range(2):
        for n, tol in (("u", 1e-12), ("v", 1e-12), ("w", 1e-12), ("p", 1e-11)):
            # launch shapes change only the block order of the mass-flux sum;
            # the forcing's last-bit change is not divergence-free after
            # rounding, and p accumulates the projection of that round-off
            assert relerr(b.channels[i].get_field(n), ref.channels[i].get_field(n)) < tol, n


def test_mixed_batch_divergence_gate():
    _need_gpu()
    from chapsim1ww_b200 import MIXED, ChannelBatch, batch64_configs
    cfgs = batch64_configs(seed=3, n=8)
    b = ChannelBatch(cfgs, precision=MIXED)
    b.init_random(seed=3, amp=0.1, project=True)
    b.step(5)
    b.sync()
    for ch in b.channels:
        assert ch.divgck_tg() <= 1e-8
        assert ch.nan_count() == 0


def test_tuned_march_is_the_one_that_runs():
    """The march length that get_tuning reports, before and after autotune, is
    the one launched: a channel that is given it explicitly leaves the same
    bits (the mass-flux sum follows the march)."""
    _need_gpu()
    from chapsim1ww_b200 import ChannelBatch, TGChannel
    b = ChannelBatch(CFGS)
    b.init_random(seed=3, amp=0.1, project=True)
    for tune in (False, True):
        if tune:
            b.autotune(reps=3)
        shapes = [c.get_tuning() for c in b.channels]
        b.init_random(seed=3, amp=0.1, project=True)
        b.step(3)
        b.sync()
        for i, c in enumerate(CFGS):
            s = TGChannel(**c)
            s.set_tuning(*shapes[i])
            s.random_fl_fld_tg(3 + i, 0.1, project=True)
            s.step(3)
            for n in ("u", "v", "w", "p"):
                assert np.array_equal(s.get_field(n), b.channels[i].get_field(n)), (tune, i, n, shapes[i])


def test_autotune_leaves_the_row_count_that_nothing_reads():
    """The register-blocked forward x transform (short lengths, and others on
    enough lines) does not read fft_lb: the autotuner has nothing to choose
    there and keeps what was set."""
    _need_gpu()
    from chapsim1ww_b200 import ChannelBatch
    cfgs = [dict(nx=n, ny=16, nz=16, ren=2500.0) for n in (10, 12, 14, 18, 20, 22)]
    cfgs += [dict(nx=n, ny=48, nz=64, ren=2500.0) for n in (60, 112)]
    b = ChannelBatch(cfgs)
    b.init_random(seed=3, amp=0.1, project=True)
    for c in b.channels:
        c.set_tuning(16, 2)
    b.autotune(reps=2)
    assert [c.get_tuning()[1] for c in b.channels] == [2] * len(cfgs)
