"""The acceptance rules of the kernels on both sides of where the engine
changes from one to the other (a moderate field, 0 < H < 2: always accepted
from 3 unsatisfied bonds for spins down and 4 for spins up; the general rule
beyond), in the resident and the streaming engine, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FIELDS = [1e-12, 0.1875, 1.0, 1.999, 2.0, 2.5, 4.0]


def _run(csg, orc, L, W, T, H, n, flags):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    seed = 31 + L
    betas = orc.geometric_betas(T, 0.3, 8.0)
    spins, bonds = orc.init(L, W, 2, T, seed)
    with csg.Engine(L, W, 2, betas, H=H, seed=seed, sweeps_per_swap=1, sweeps_per_meas=1,
                    flags=csg.CSG_MEASURE_M | flags, swap_log_rounds=n) as e:
        e.set_state(spins, bonds, 0)
        e.run(n)
        s_gpu, _, _ = e.get_state()
        o = e.observables()
    want = orc.Observables(L, W, 2, T, log_rounds=n)
    orc.run(spins, bonds, L=L, betas=betas, H=H, seed=seed, sweep0=0, n_sweeps=n, sweeps_per_swap=1,
            sweeps_per_meas=1, obs=want)
    np.testing.assert_array_equal(s_gpu, spins)
    for f in ("e_sum", "m_sum", "e_last", "m_last", "q2_sum", "d_last", "swap_acc", "swap_log"):
        np.testing.assert_array_equal(getattr(o, f), getattr(want, f), err_msg=f)


@pytest.mark.parametrize("H", FIELDS)
def test_resident_rule(csg, orc, H):
    _run(csg, orc, 12, 1, 8, H, 8, 0)


@pytest.mark.parametrize("H", [1e-12, 1.999, 2.0, 4.0])
@pytest.mark.parametrize("L", [8, 20])
def test_resident_rule_sizes(csg, orc, L, H):
    _run(csg, orc, L, 1, 4, H, 4, 0)


@pytest.mark.parametrize("H", FIELDS)
def test_streaming_rule(csg, orc, H):
    _run(csg, orc, 10, 2, 8, H, 6, csg.CSG_ENGINE_STREAM)
