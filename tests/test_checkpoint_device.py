"""Checkpoint conversion on the device: the state of a checkpoint, word for
word, against a numpy restatement of the layout; the error a damaged one
gives (the first violation in the order words, sites, samples; copies before
ends of a bond) and the state it leaves; and more words than one upload holds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _need_gpu():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _ref(L, W, T, seed):
    rng = np.random.default_rng(seed)
    S = 32 * W
    v = rng.integers(0, 1 << T, (S, 2, L, L, L), dtype=np.uint32)
    bond = rng.integers(0, 2, (3, S, 1, L, L, L), dtype=np.uint32)  # 1: ferromagnetic
    for k in range(3):
        v |= (bond[k] << np.uint32(27 + 2 * k)) | (np.roll(bond[k], 1, axis=4 - k) << np.uint32(26 + 2 * k))
    return v.reshape(2 * S, L ** 3), bond[:, :, 0]


def _pack(bits, axis):
    """32 samples of a word as the bits of a uint32."""
    sh = np.arange(32, dtype=np.uint32)
    return np.bitwise_or.reduce(bits.astype(np.uint32) << sh.reshape([-1] + [1] * (bits.ndim - axis - 1)), axis=axis)


def _state(ref, bond, L, W, T):
    N = L ** 3
    z, y, x = np.meshgrid(*[np.arange(L)] * 3, indexing="ij")
    slot = (((x + y + z) & 1) * (N // 2) + (z * L + y) * (L // 2) + x // 2).reshape(-1)
    v = ref.reshape(W, 32, 2, N)
    spins = np.zeros((W, 2, T // 4, N, 4), np.uint32)
    for t in range(T):
        spins[:, :, t // 4, slot, t % 4] = _pack((v >> np.uint32(t)) & 1, 1)
    bonds = np.zeros((W, 3, N), np.uint32)
    for k in range(3):
        bonds[:, k, slot] = _pack(1 - bond[k].reshape(W, 32, N), 1)
    return spins, bonds


@pytest.mark.parametrize("L,W,T", [(4, 1, 4), (6, 3, 24), (10, 2, 12), (26, 1, 8)])
def test_checkpoint_is_the_packed_state(csg, L, W, T):
    ref, bond = _ref(L, W, T, L + T)
    with csg.Engine(L, W, 2, np.linspace(2.0, 0.5, T), seed=1) as e:
        e.load_checkpoint(ref, 7)
        spins, bonds, sweep = e.get_state()
        want_s, want_b = _state(ref, bond, L, W, T)
        np.testing.assert_array_equal(spins, want_s)
        np.testing.assert_array_equal(bonds, want_b)
        assert sweep == 7
        np.testing.assert_array_equal(e.save_checkpoint(), ref)


def test_damaged_checkpoints(csg):
    L, W, T = 6, 2, 8
    ref, _ = _ref(L, W, T, 3)
    N = L ** 3
    ends, copies = ref.copy(), ref.copy()
    # sample 40, site 100: the -z bond of both copies (still alike, but not what
    # the other end says); sample 33, site 7: one copy only, met first
    ends[2 * 40:2 * 40 + 2, 100] ^= np.uint32(1 << 30)
    copies[2 * 40:2 * 40 + 2, 100] ^= np.uint32(1 << 30)
    copies[2 * 33 + 1, 7] ^= np.uint32(1 << 26)
    with csg.Engine(L, W, 2, np.linspace(2.0, 0.5, T), seed=5) as e:
        e.load_checkpoint(ref, 11)
        for bad, words in ((ends, "two ends"), (copies, "copies")):
            with pytest.raises(csg.CsgError) as err:
                e.load_checkpoint(bad, 0)
            assert err.value.code == 4 and words in str(err.value)
        with pytest.raises(csg.CsgError) as err:
            e.load_checkpoint(ref, -1)
        assert err.value.code == 1
        np.testing.assert_array_equal(e.save_checkpoint(), ref)  # as it was
        assert e.get_state()[2] == 11


def test_more_words_than_one_upload(csg):
    L, W, T = 40, 17, 4  # 16.4 MB a word, 16 of them at once
    rng = np.random.default_rng(9)
    with csg.Engine(L, W, 2, np.linspace(2.0, 0.5, T), seed=6) as e:
        e.init_lattice()
        spins, bonds, _ = e.get_state()
        ref = e.save_checkpoint()
        e.set_state(rng.integers(0, 1 << 32, spins.shape, dtype=np.uint32), bonds, 0)
        e.load_checkpoint(ref, 3)
        s2, b2, sweep = e.get_state()
        assert sweep == 3
        np.testing.assert_array_equal(s2, spins)
        np.testing.assert_array_equal(b2, bonds)
        ref[-1, 5] ^= np.uint32(1 << 27)  # the last word, past the first upload
        with pytest.raises(csg.CsgError):
            e.load_checkpoint(ref, 0)
