"""The integers of the observable records (bonds, spins up, differing sites per
coordinate plane), through the records they give, where the kernels' shapes
change: the smallest lattice, planes that are not whole warps, every size of
the lanes' counters, several blocks per quad.  The reference's definitions on
the state, in doubles, against floats: 1e-6 of values up to 3."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("L,W,T", [(4, 1, 4), (6, 2, 8), (10, 1, 4), (14, 1, 12), (22, 1, 4), (26, 1, 4), (46, 1, 4)])
def test_records_of_a_random_state(csg, L, W, T):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    N, H = L ** 3, 0.25
    rng = np.random.default_rng(L)
    z, y, x = np.meshgrid(*[np.arange(L)] * 3, indexing="ij")
    slot = ((x + y + z) & 1) * (N // 2) + (z * L + y) * (L // 2) + x // 2
    with csg.Engine(L, W, 2, np.linspace(2.0, 0.5, T), H=H, seed=1) as e:
        spins = rng.integers(0, 1 << 32, e.spin_shape, dtype=np.uint32)
        spins[:, 1] = np.where(rng.random(spins[:, 1].shape) < 0.7, spins[:, 0], spins[:, 1])
        bonds = rng.integers(0, 1 << 32, e.bond_shape, dtype=np.uint32)
        e.set_state(spins, bonds, 0)
        rec = e.obs_records()
        again = e.obs_records()
    np.testing.assert_array_equal(rec, again)
    wave = np.exp(2j * np.pi * np.arange(L) / L)
    for w in range(W):
        for b in (0, 13, 31):
            J = 1.0 - 2.0 * ((bonds[w][:, slot] >> np.uint32(b)) & 1)
            for t in range(T):
                s = [2.0 * ((spins[w, c, t // 4, :, t % 4][slot] >> np.uint32(b)) & 1) - 1.0 for c in (0, 1)]
                want = np.zeros(11)
                for c in (0, 1):
                    bond = sum((J[k] * s[c] * np.roll(s[c], -1, axis=2 - k)).sum() for k in range(3))
                    want[c], want[2 + c] = -(bond + H * s[c].sum()) / N, s[c].sum() / N
                q = s[0] * s[1]
                want[4] = q.sum() / N
                for k in range(3):
                    f = (q.sum(axis=tuple(i for i in range(3) if i != 2 - k)) * wave).sum() / N
                    want[5 + k], want[8 + k] = f.real, f.imag
                np.testing.assert_allclose(rec[32 * w + b, t], want, atol=1e-6, err_msg=f"{w} {b} {t}")


@pytest.mark.gpu
@pytest.mark.parametrize("L", [6, 12, 22])
def test_records_of_spins_off_a_16_byte_boundary(csg, L):
    """csg_obs_records_noalloc takes spins at any 4-byte address."""
    import ctypes as C
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    f = csg.lib().csg_obs_records_noalloc
    f.argtypes = [C.POINTER(csg.Config), C.c_void_p, C.c_void_p, C.c_void_p, C.c_size_t, C.c_void_p]
    W, T = 1, 8
    with csg.Engine(L, W, 2, np.linspace(2.0, 0.5, T), seed=3) as e:
        e.init_lattice()
        want = e.obs_records()
        s, b, _ = e.get_state()
        db = torch.from_numpy(b.view(np.int32).reshape(-1)).cuda()
        for off in (0, 1, 2, 3):
            ds = torch.zeros(s.size + 4, dtype=torch.int32, device="cuda")
            ds[off:off + s.size] = torch.from_numpy(s.view(np.int32).reshape(-1))
            out = torch.zeros((32 * W, T, 11), device="cuda")
            assert f(C.byref(e.cfg), ds.data_ptr() + 4 * off, db.data_ptr(), out.data_ptr(), out.numel(),
                     torch.cuda.current_stream().cuda_stream) == 0
            torch.cuda.synchronize()
            np.testing.assert_array_equal(out.cpu().numpy(), want)
