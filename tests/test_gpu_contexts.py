"""Contexts of different sizes in one process, from one host thread and from
several: the kernels' limits on dynamic shared memory belong to the library,
so no context may change what another one's launches need."""
import threading

import numpy as np
import pytest

from _util import channel_state, config0_params, grid_for

pytestmark = pytest.mark.gpu

# 32 modes a CTA in both column solves (105 to 211 KB for the CN solve), and
# 8 modes (109 to 226 KB), each at two lengths of the columns
SIZES = {"wide": [(128, 33, 128), (128, 80, 128)], "long": [(32, 110, 32), (32, 250, 32)]}


def channels(sizes, prec=0):
    from diablo3_b200.channel import Channel
    out = []
    for n in sizes:
        p = config0_params(nx=n[0], ny=n[1], nz=n[2], precision=prec)
        ch = Channel(p, grid_for(p))
        ch.init_flow(seed=3)
        out.append((p, ch))
    return out


def substeps(ch, n):
    for k in range(n):
        ch.rk_chan_1(1 + k % 3)


def alone(sizes, drive, prec=0):
    out = []
    for p, ch in channels(sizes, prec):
        with ch:
            drive(ch)
            out.append(channel_state(ch, p))
    return out


def same(got, want):
    return all(np.array_equal(g[f], w[f]) for g, w in zip(got, want) for f in w)


@pytest.mark.parametrize("sizes", SIZES)
@pytest.mark.parametrize("prec", [0, 1])
def test_channels_of_two_sizes_step_in_turn(sizes, prec):
    """Replayed step graphs and direct substeps of a long channel after a short one's."""
    want = alone(SIZES[sizes], lambda ch: (ch.step(2), substeps(ch, 3)), prec)
    pairs = channels(SIZES[sizes], prec)
    for _ in range(2):
        for _, ch in reversed(pairs):
            ch.step(1)
    for k in range(3):
        for _, ch in pairs[::1 if k % 2 else -1]:
            ch.rk_chan_1(1 + k)
    assert same([channel_state(ch, p) for p, ch in pairs], want)
    for _, ch in pairs:
        ch.close()


@pytest.mark.parametrize("sizes", SIZES)
def test_channels_of_two_sizes_on_two_threads(sizes):
    """One host thread per context, as the C-ABI allows: 300 substeps each, launched side by side."""
    want = alone(SIZES[sizes], lambda ch: substeps(ch, 300))
    pairs = channels(SIZES[sizes])
    start, errs = threading.Barrier(len(pairs)), []

    def work(ch):
        try:
            start.wait()
            substeps(ch, 300)
        except Exception as e:   # noqa: BLE001 - reported below
            errs.append(e)

    th = [threading.Thread(target=work, args=(ch,)) for _, ch in pairs]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not errs, errs
    assert same([channel_state(ch, p) for p, ch in pairs], want)
    for _, ch in pairs:
        ch.close()


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n", [(128, 63, 64), (64, 33, 128)])
def test_equal_members_stay_equal(n, prec):
    """24 members with one state: 60 steps later every bit is still the same in all of them."""
    from diablo3_b200.ensemble import Ensemble
    p = config0_params(nx=n[0], ny=n[1], nz=n[2], precision=prec)
    ens = Ensemble([p] * 24, grid_for(p), init=False)
    ens.members[0].init_flow(seed=3)
    state = ens.members[0].download_state()
    for m in ens.members:
        m.upload_state(state)
    ens.step(60)
    first = channel_state(ens.members[0], p)
    for m in ens.members[1:]:
        s = channel_state(m, p)
        assert all(np.array_equal(s[f], first[f]) for f in s)
    ens.close()
