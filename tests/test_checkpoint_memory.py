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


def test_checkpoints_on_a_full_device(csg):
    """No room for a single word's scratch: the conversion runs in host memory."""
    import torch
    L, W, T = 46, 2, 8  # 24.9 MB a word
    betas = np.linspace(2.0, 0.5, T)
    with csg.Engine(L, W, 2, betas, seed=8) as e:
        e.init_lattice()
        want_s, want_b, _ = e.get_state()
        ref = e.save_checkpoint()  # also loads the kernels
        e.load_checkpoint(ref, 1)
        csg.trim_scratch()
        torch.cuda.empty_cache()
        filler = []
        size = 1 << 36
        while size >= 1 << 21:  # less than one of torch's segments of 20 MB is left
            try:
                filler.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
            except torch.cuda.OutOfMemoryError:
                size //= 2
        try:
            assert torch.cuda.mem_get_info()[0] < 64 * L ** 3 * 4
            np.testing.assert_array_equal(e.save_checkpoint(), ref)
            e.set_state(np.zeros_like(want_s), np.zeros_like(want_b), 0)
            e.load_checkpoint(ref, 9)
            bad = ref.copy()
            bad[-1, 5] ^= np.uint32(1 << 27)
            with pytest.raises(csg.CsgError, match="copies"):
                e.load_checkpoint(bad, 0)
        finally:
            del filler
            torch.cuda.empty_cache()
        spins, bonds, sweep = e.get_state()
    assert sweep == 9
    np.testing.assert_array_equal(spins, want_s)
    np.testing.assert_array_equal(bonds, want_b)
