"""The chunked column solves (k_cn_solve, k_rem_div_ch) at the edges of their
chunks and of the forms the launcher picks: 32 chunks of 8 modes (small
planes) or of 4 (long columns), 16 of 16 and 8 of 32 (larger planes), and the
one-thread-per-mode kernels where the columns leave shared memory."""
import pytest

from _util import NAMES, STATE, channel_state, config0_params, grid_for, oracle_state, rel_l2, seed_pair

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [
    (16, 4, 16), (16, 29, 16), (16, 30, 32), (16, 31, 16), (32, 62, 16), (16, 63, 16),   # 32 chunks of 8 modes
    (16, 262, 16), (16, 263, 16),             # 8 -> 4 modes a CTA in the CN solve
    (16, 398, 16), (16, 399, 16),             # the CN solve back on the two kernels
    (128, 14, 64), (128, 15, 64),             # 16 chunks of 16 modes
    (128, 5, 128), (128, 6, 128), (128, 7, 128), (128, 88, 128),   # 8 chunks of 32 modes
])
def test_step_matches_oracle(oracle_mod, n):
    from diablo3_b200.channel import Channel
    nx, ny, nz = n
    p = config0_params(nx=nx, ny=ny, nz=nz)
    o, ch = seed_pair(oracle_mod.Oracle, Channel, p, grid_for(p), seed=5)
    with ch:
        o.step()
        ch.step(1)
        so, sg = oracle_state(o, p), channel_state(ch, p)
        errs = {NAMES[f]: rel_l2(sg[f], so[f]) for f in STATE}
        # the suite's FP64 bar.  cp after one step is phi / h of a projection of
        # d u2 / dy, whose round-off grows as 1 / dy ~ ny (6e-12 at ny 65, up to
        # 2.1e-10 at ny 399, the same with one thread per column): 2.5e-12 ny
        cp = errs.pop("cp")
        assert all(v <= 1e-10 for v in errs.values()) and cp <= max(1e-10, 2.5e-12 * ny), (errs, cp)
        # round-off of d u2 / dy: 2e-16 over the finest spacing (2e-3 at ny 399), a few tens of roundings
        assert ch.divergence() <= 1e-11
