"""The streaming engine's colour launches (a thread walks a chunk of z-planes)
where their shapes can go wrong: a plane that is not whole blocks, chunks that
do not tile the lattice, one quad alone (the shortest chunks) and enough of
them for the longest, one copy and both, with and without counters."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# L, W, C, T, H, sweeps, sps, spm, M
CASES = [
    (34, 1, 1, 4, 0.0, 3, 0, 0, False),   # updates only, one quad
    (38, 1, 2, 4, 0.0, 3, 0, 1, True),    # measurement without exchange, magnetisations
    (26, 6, 2, 32, 0.0, 2, 1, 0, False),  # many quads, exchange without measurement
    (36, 3, 1, 12, 0.0, 3, 2, 1, True),
    (42, 1, 2, 8, 0.4, 2, 1, 1, False),
    (6, 1, 2, 4, 0.0, 9, 2, 3, False),    # the walk longer than the lattice (forced)
]


@pytest.mark.parametrize("L,W,C_,T,H,n,sps,spm,M", CASES)
def test_colour_walk_matches_oracle(csg, orc, L, W, C_, T, H, n, sps, spm, M):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    seed = 77 + L
    betas = orc.geometric_betas(T, 0.4, 2.0)
    spins, bonds = orc.init(L, W, C_, T, seed)
    flags = csg.CSG_ENGINE_STREAM | (csg.CSG_MEASURE_M if M else 0)
    rounds = n // sps if sps else 0
    with csg.Engine(L, W, C_, betas, H=H, seed=seed, sweeps_per_swap=sps, sweeps_per_meas=spm,
                    flags=flags, swap_log_rounds=max(rounds, 1)) as e:
        e.set_state(spins, bonds, 0)
        e.run(n)
        s_gpu, _, _ = e.get_state()
        o_gpu = e.observables()
    o_orc = orc.Observables(L, W, C_, T, log_rounds=max(rounds, 1))
    orc.run(spins, bonds, L=L, betas=betas, H=H, seed=seed, sweep0=0, n_sweeps=n, sweeps_per_swap=sps,
            sweeps_per_meas=spm, obs=o_orc)
    np.testing.assert_array_equal(s_gpu, spins)
    assert o_gpu.n_meas == o_orc.n_meas and o_gpu.boundary == 0
    fields = ["e_sum", "e_last", "swap_acc"] + (["m_sum", "m_last"] if M else [])
    fields += ["q_sum", "q2_sum", "q4_sum", "hist", "d_last"] if C_ == 2 else []
    for f in fields:
        np.testing.assert_array_equal(getattr(o_gpu, f), getattr(o_orc, f), err_msg=f)
    if rounds:
        np.testing.assert_array_equal(o_gpu.swap_log[:rounds], o_orc.swap_log[:rounds])
