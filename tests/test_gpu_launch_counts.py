"""The launch counter (db_kernel_launches, db_ensemble_info) against the kernels
of a step, one by one, in every form of the substep."""
import ctypes

import pytest

from _util import config0_params, grid_for

pytestmark = pytest.mark.gpu

TRI, REM = 2, 1                       # rows and elimination of the implicit systems; projection
PHYS, PROD = 2, 1                     # z and x to physical space; products with their x-pass
CFL = 3 + 1                           # two passes and the minimum, dt applied
LES_CFL = 2 + 1                       # reduction and the minimum, dt applied
MODEL = 2                             # ghost rows, closure
BACK = 1 + 1 + 2                      # x to physical, eddy-viscosity solves, x and z to Fourier space


@pytest.mark.parametrize("kw, substep, extra", [
    (dict(nx=16, ny=17, nz=16), TRI + PHYS + PROD + 1 + 1 + REM, 0),
    (dict(nx=16, ny=17, nz=16, precision=1), TRI + PHYS + PROD + 1 + 1 + REM, 0),
    (dict(nx=16, ny=17, nz=16, variable_dt=1), TRI + PHYS + PROD + 1 + 1 + REM, CFL),
    (dict(nx=16, ny=400, nz=16), TRI + PHYS + PROD + 1 + 2 + REM, 0),     # the CN solve in two kernels
    (dict(nx=512, ny=5, nz=512), TRI + PHYS + PROD + 1 + 2 + REM, 0),
    (dict(nx=16, ny=17, nz=16, use_les=1, create_new_flow=0), TRI + MODEL + PHYS + PROD + 3 + BACK + REM, 0),
    (dict(nx=32, ny=17, nz=16, use_les=1, create_new_flow=0, precision=1, variable_dt=1),
     TRI + MODEL + PHYS + PROD + 1 + BACK + REM, LES_CFL),
])
def test_launches_of_a_step(kw, substep, extra):
    from diablo3_b200.channel import Channel
    p = config0_params(**kw)
    with Channel(p, grid_for(p)) as ch:
        n = ctypes.c_longlong()
        for k in (1, 2):                # captured, replayed
            ch.step(1)
            ch._ck(ch.L.db_kernel_launches(ch.h, ctypes.byref(n)))
            assert n.value == k * (2 + 3 * substep + extra)


@pytest.mark.parametrize("ny, cn", [(17, 1), (400, 2)])
def test_launches_of_a_batched_step(ny, cn):
    from diablo3_b200.ensemble import Ensemble
    p = config0_params(nx=16, ny=ny, nz=16)
    ens = Ensemble([p, p], grid_for(p), init=False)
    ens.step(1)
    assert ens.batched and ens.kernels_per_step() == 2 + 3 * (TRI + PHYS + PROD + 1 + cn + REM)
    ens.close()
