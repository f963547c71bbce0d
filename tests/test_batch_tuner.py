"""The batch tuner weighs the plan every member starts from: where the GPU is
not full that is a larger team than the splits tried on a full one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2])  # members alike: each of them bounds the batch
def test_tuned_batch_keeps_the_planned_team(csg, n):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    members = [dict(L=12, n_words=1, n_copies=2, betas=np.linspace(2.0, 0.5, 16), seed=3 + i, sweeps_per_swap=16)
               for i in range(n)]
    with csg.Batch(members) as b:
        for e in b.members:
            e.init_lattice()
        # one word at L = 12: 432 threads a quad take 3.1 us a sweep; the splits for a
        # full GPU have 144 at most, 4.2 us
        for _ in range(2):  # the second time from the plans of the first
            assert [b.member_plan(i).threads_per_quad for i in range(n)] == [432] * n
            b.tune(256)
        assert [b.member_plan(i).threads_per_quad for i in range(n)] == [432] * n
