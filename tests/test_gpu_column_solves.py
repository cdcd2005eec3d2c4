"""The column solves (k_cn_solve, k_rem_div_ch and the one-thread-per-mode
k_rhs_cn, k_cn_back, k_rem_div) at the edges of their chunks and of the forms
the launchers pick, on both work types."""
import pytest

from _util import NAMES, channel_state, config0_params, grid_for, oracle_state, rel_l2, seed_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n", [
    (16, 4, 16), (16, 29, 16), (16, 30, 32), (16, 31, 16), (32, 62, 16), (16, 63, 16),   # 32 chunks of 8 modes
    (16, 262, 16), (16, 263, 16),             # 8 -> 4 modes a CTA in the CN solve
    (16, 398, 16), (16, 399, 16),             # the CN solve on its two kernels
    (16, 881, 16), (16, 882, 16),             # the projection one thread per column, four rows in flight
    (32, 30, 128), (32, 31, 128), (32, 96, 128), (32, 97, 128),   # 1020 modes: 8 -> 16 chunks; projection 16 -> 32
    (128, 14, 64), (128, 30, 64), (128, 31, 64), (128, 62, 64), (128, 63, 64),   # 1892 modes: 4 -> 8 -> 16 chunks
    (128, 5, 128), (128, 7, 128), (128, 88, 128), (128, 89, 128),  # 3740 modes: 4, 8 and (shared memory) 16 chunks
    (512, 5, 512), (512, 9, 512),             # more modes than the chunked forms take: two kernels, three rows in flight
])
def test_step_matches_oracle(oracle_mod, n, prec):
    from diablo3_b200.channel import Channel
    nx, ny, nz = n
    p = config0_params(nx=nx, ny=ny, nz=nz, precision=prec)
    o, ch = seed_pair(oracle_mod.Oracle, Channel, p, grid_for(p), seed=5)
    with ch:
        o.step()
        ch.step(1)
        so, sg = oracle_state(o, p), channel_state(ch, p)
        # FP64: all nine fields.  Mixed: the state; the history holds the
        # FP32 nonlinear terms themselves (test_gpu_mixed.py)
        errs = {NAMES[f]: rel_l2(sg[f], so[f]) for f in ((0, 1, 2, 3, 4) if prec else range(9))}
        cp = errs.pop("cp")
        if prec:
            # FP32 round-off (6e-8) of terms that change the state by dt = 1e-3 of
            # themselves: 1e-10 times a few roundings; cp takes it undivided
            assert all(v <= 1e-8 for v in errs.values()) and cp <= 1e-5, (errs, cp)
        else:
            # the suite's FP64 bar.  cp after one step is phi / h of a projection of
            # d u2 / dy, whose round-off grows as 1 / dy ~ ny (6e-12 at ny 65, up to
            # 2.1e-10 at ny 399, the same with one thread per column): 2.5e-12 ny
            assert all(v <= 1e-10 for v in errs.values()) and cp <= max(1e-10, 2.5e-12 * ny), (errs, cp)
        assert ch.divergence() <= 1e-12


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n", [
    (16, 31, 16), (16, 263, 16), (16, 399, 16), (128, 15, 64), (128, 31, 64), (128, 63, 64), (512, 5, 512)])
def test_batched_forms_give_the_bits_of_solo_runs(n, prec):
    """Each form of the column solves with the member index folded in: 32 chunks of 8 and of 4 modes, two kernels,
    4, 8 and 16 chunks, and the planes the chunked forms leave out."""
    import numpy as np
    from diablo3_b200.channel import Channel
    from diablo3_b200.ensemble import Ensemble
    ps = [config0_params(nx=n[0], ny=n[1], nz=n[2], precision=prec, dthdx_override=m2) for m2 in (0.8, 1.2)]
    gy = grid_for(ps[0])
    ens = Ensemble(ps, gy, seeds=[3, 4])
    assert ens.batched
    ens.step(2)
    for p, m, seed in zip(ps, ens.members, (3, 4)):
        with Channel(p, gy) as ch:
            ch.init_flow(seed=seed)
            ch.step(2)
            a, b = channel_state(m, p), channel_state(ch, p)
            assert all(np.array_equal(a[f], b[f]) for f in a)
    ens.close()
