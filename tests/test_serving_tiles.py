"""Requests that share the GPU take smaller tiles while SMs are free, the one
that would finish last first: whatever tiles a mix gives a request, its result
is the one it has alone."""
import numpy as np
import pytest

# L, words, temperatures, sweeps
MIXES = [
    [(8, 1, 12, 70), (12, 1, 16, 40), (16, 1, 24, 30)],                 # few quads: the smallest tiles
    [(10, 9, 24, 40), (14, 6, 20, 20), (16, 8, 24, 20), (6, 3, 8, 90)],  # about as many CTAs as SMs
    [(16, 40, 24, 4), (12, 2, 8, 50), (26, 1, 4, 6)],                    # a full GPU, and a streamed lattice
]


@pytest.mark.gpu
@pytest.mark.parametrize("mix", MIXES)
def test_mixed_requests_equal_alone(csg, mix):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    kw = [dict(L=L, n_words=W, n_copies=2, betas=csg.geometric_betas(T, 0.3, 2.0), seed=50 + i, sweeps_per_swap=1,
               sweeps_per_meas=2) for i, (L, W, T, _) in enumerate(mix)]
    with csg.Server(8 << 30, 8, 16) as srv:
        ids = [srv.submit(n, **k) for k, (_, _, _, n) in zip(kw, mix)]
        got = {}
        while len(got) < len(ids):
            for i in srv.poll()[0]:
                got[i] = srv.result(i, with_spins=True)
    for i, k, (_, _, _, n) in zip(ids, kw, mix):
        with csg.Engine(**k) as e:
            e.init_lattice()
            e.run(n)
            spins, _, _ = e.get_state()
            o = e.observables()
        np.testing.assert_array_equal(got[i][1], spins)
        for f in ("e_sum", "q_sum", "q2_sum", "q4_sum", "hist", "e_last", "d_last", "swap_acc"):
            np.testing.assert_array_equal(getattr(got[i][0], f), getattr(o, f), err_msg=f)
