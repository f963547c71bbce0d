"""Whose memory the checkpoint calls use, and until when, on the device."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _need_gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def test_a_page_locked_checkpoint_may_be_overwritten_after_the_load(csg):
    import torch
    L, W, T = 40, 17, 4  # more words than one upload holds
    betas = np.linspace(2.0, 0.5, T)
    with csg.Engine(L, W, 2, betas, seed=6) as e:
        e.init_lattice()
        want_s, want_b, _ = e.get_state()
        pinned = torch.empty((64 * W, L ** 3), dtype=torch.int32, pin_memory=True)
        ref = pinned.numpy().view(np.uint32)
        ref[:] = e.save_checkpoint()
        e.set_state(np.zeros_like(want_s), want_b, 0)
        e.load_checkpoint(ref, 3)
        ref[:] = 0
        spins, bonds, sweep = e.get_state()
    assert sweep == 3
    np.testing.assert_array_equal(spins, want_s)
    np.testing.assert_array_equal(bonds, want_b)
