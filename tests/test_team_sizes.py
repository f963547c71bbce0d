"""Teams of the resident kernel with many threads per quad (short column
segments), which the planner takes where an SM has few quads: every built split
with one quad per CTA and with as many as fit, against the oracle; and the
planner's choice for a simulation that fills few SMs."""
import numpy as np
import pytest

# L, column segments per thread
SPLITS = [(6, 6), (8, 4), (8, 8), (10, 5), (12, 4), (12, 6), (16, 4), (18, 3), (20, 2)]


def _need_gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _check(csg, orc, L, W, C_, T, H, n):
    seed = 400 + L
    betas = orc.geometric_betas(T, 0.4, 2.5)
    spins, bonds = orc.init(L, W, C_, T, seed)
    with csg.Engine(L, W, C_, betas, H=H, seed=seed, sweeps_per_swap=1, sweeps_per_meas=1,
                    flags=csg.CSG_MEASURE_M, swap_log_rounds=n) as e:
        e.set_state(spins, bonds, 0)
        e.run(n)
        s_gpu, _, _ = e.get_state()
        o = e.observables()
    want = orc.Observables(L, W, C_, T, log_rounds=n)
    orc.run(spins, bonds, L=L, betas=betas, H=H, seed=seed, sweep0=0, n_sweeps=n, sweeps_per_swap=1,
            sweeps_per_meas=1, obs=want)
    np.testing.assert_array_equal(s_gpu, spins)
    fields = ["e_sum", "m_sum", "e_last", "m_last", "swap_acc", "swap_log"]
    fields += ["q_sum", "q2_sum", "q4_sum", "hist", "d_last"] if C_ == 2 else []
    for f in fields:
        np.testing.assert_array_equal(getattr(o, f), getattr(want, f), err_msg=f)


@pytest.mark.gpu
@pytest.mark.parametrize("H", [0.0, 0.4, 2.5])
@pytest.mark.parametrize("L,nseg", SPLITS)
def test_every_split_matches_oracle(csg, orc, L, nseg, H):
    _need_gpu()
    tpq = L * (L // 2) * nseg
    try:
        for qc in (1, 2, 4):
            if qc * tpq > 512 or qc * L ** 3 * 16 > 200 * 1024:
                continue
            csg.set_plan_override(qc, tpq)
            _check(csg, orc, L, 1, 2, 8, H, 5)
    finally:
        csg.set_plan_override(None)


@pytest.mark.gpu
def test_short_columns_where_the_gpu_is_not_full(csg, orc):
    _need_gpu()
    # one word: a quad per CTA and the largest team; a full GPU: the default team
    # (a smaller one where every sweep also reduces)
    p = csg.query_plan(12, 1, 2, np.linspace(2.0, 0.5, 16), sweeps_per_swap=16)
    assert (p.quads_per_cta, p.threads_per_quad) == (1, 432)
    p = csg.query_plan(12, 1, 2, np.linspace(2.0, 0.5, 16))
    assert (p.quads_per_cta, p.threads_per_quad) == (1, 288)
    p = csg.query_plan(16, 32, 2, np.linspace(2.0, 0.5, 24))
    assert (p.quads_per_cta, p.threads_per_quad) == (3, 128)
    # planned again from what was kept: the same, and the override still decides
    assert csg.query_plan(12, 1, 2, np.linspace(2.0, 0.5, 16)).threads_per_quad == 288
    csg.set_plan_override(2, 144)
    try:
        p = csg.query_plan(12, 1, 2, np.linspace(2.0, 0.5, 16))
        assert (p.quads_per_cta, p.threads_per_quad) == (2, 144)
    finally:
        csg.set_plan_override(None)
    _check(csg, orc, 12, 1, 1, 4, 0.0, 4)
